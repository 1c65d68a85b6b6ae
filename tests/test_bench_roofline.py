"""What the bench says of the partitioned dual CG: no fraction of a rate that it
does not use."""

import bench as B


def test_no_hbm_fraction_for_the_partitioned_kernel():
  nv, nt, n2 = 68921, 718520, 398520
  ne = 4 * (nt - n2) + 2 * n2
  st = [dict(ms_warm=7.6, ms_dual=50.0, cg_iters_warm=56, cg_iters_total=770, cg_launches=2, newton_iters=1,
             cg_path='primal')] * 2
  r = B.roofline_of_solver(st, nt, nv, 8, 6701.2, 'measured', 40, 'edge_volume', (ne, n2))
  d, p = (r, r['other']) if r['kernel'].startswith('k_dcg') else (r['other'], r)
  assert d['kernel'].startswith('k_dcg') and p['kernel'].startswith('k_pcg')
  assert d['frac'] is None and d['peak'] is None and d['achieved'] is None and d['traffic'] is None
  assert 'dram_frac' not in d and 'cg_path' not in d
  assert d['bound'] == 'exchange between blocks'
  assert d['meetings_per_cg_iteration'] == 10
  assert abs(d['us_per_meeting'] - 50.0e3 / 714 / 10) <= 0.01
  # the primal kernel keeps its own line
  assert p['bound'] == 'hbm' and p['frac'] > 0
