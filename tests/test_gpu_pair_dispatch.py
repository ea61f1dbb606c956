"""The instantiations that large grids take, against the FP64 oracle at the parity
bar (relative L2 <= 1e-4 of every wavefield): thin grids with one long axis that
still cross the thresholds of the dispatch.  The tiles the launches take are
asserted, so a threshold that moves cannot move a case to another kernel unseen.

* the stress kernels with eight rows at 256 points, and with a last tile of two
  and of six rows, whose second quad is empty or half inside the grid, where the
  mirror points come by shuffle (64 and 96 points) and by a second load (120);
* the velocity kernels with 32 z per block at 256 points;
* three-stage lengths above 256 on each axis."""
import pytest

import qvti_cases as qc
from test_gpu_pair_kernels import _case
from test_gpu_parity import TOL

pytestmark = pytest.mark.gpu


def _run(qvti, oracle, n, pml, vti, nt, want):
    c = _case(n, pml, seed=sum(n))
    with qvti.simulation_for_case(c, vti=vti) as sim:
        tiles, runtime = sim.tiles()
    for kernel, tile in want.items():
        assert not runtime[kernel] and tiles[kernel] == tile, (tiles, runtime)
    ours = qvti.run_case(c, nt=nt, vti=vti, src_type=0, ref_offset=False, want_state=True)
    ref = oracle.run_case(c, nt=nt, vti=vti, src_type=0, ref_offset=False, want_state=True)
    for f, name in enumerate(qvti.FIELDS):
        e = qc.relL2(ours["state"][f], ref["state"][f])
        assert e <= TOL, "%s %s relL2 %.3g" % (n, name, e)


VY, VX, SIGMA = 0, 1, 5


@pytest.mark.parametrize("n,vti", [
    ((80, 64, 256), True),    # 16 lanes of two pencils
    ((120, 42, 64), False),   # ny % 8 == 2, 8 lanes
    ((120, 42, 96), True),    # ny % 8 == 2, 8 threads for 6 butterflies
    ((100, 54, 120), True),   # ny % 8 == 6, second load
])
def test_eight_row_stress_kernels(qvti, oracle, n, vti):
    _run(qvti, oracle, n, 5, vti, 16, {SIGMA: 8})


@pytest.mark.parametrize("n,want", [((56, 256, 128), {VY: 32}), ((256, 56, 128), {VX: 32})])
def test_velocity_kernels_of_32_z(qvti, oracle, n, want):
    _run(qvti, oracle, n, 5, True, 12, want)


@pytest.mark.parametrize("n", [(320, 24, 36), (24, 360, 40), (36, 24, 384), (512, 24, 36), (24, 512, 36), (40, 36, 324)])
def test_three_stages_above_256(qvti, oracle, n):
    _run(qvti, oracle, n, 5, True, 16, {})
