"""The packed kernels (k_dv, k_st, k_dz) where they can go wrong, against the
FP64 oracle at the parity bar (relative L2 <= 1e-4): rows that are only 8-byte
aligned and a partial z quad (nz % 4 == 2), a last y tile of two rows
(ny % 4 == 2), an odd C-PML width (a row pair half inside the y slab), two- and
three-stage plans of every radix, butterflies that take their mirror points by
shuffle (a pencil of 8 or 16) and by a second load, the isotropic branch and
both sources.  Compared are the wavefields: in so few steps the wave does not
reach the receivers, and what they record is the rounding of either side."""
import numpy as np
import pytest

import qvti_cases as qc
from test_gpu_parity import TOL

pytestmark = pytest.mark.gpu

NT = 36


def _case(n, pml, seed):
    c = qc.heterogeneous_case(n=n, pml=pml, d=(10.0, 11.0, 9.0), dt=0.7e-3, nt=NT, f0=30.0, seed=seed,
                              src=(n[0] // 2, n[1] // 2, n[2] // 2), r_iz=pml + 1, name="pair")
    rng = np.random.default_rng(seed)
    c["eps"] = (0.2 * rng.random(n)).astype(np.float32)
    c["delta"] = (0.1 * rng.random(n)).astype(np.float32)
    return c


@pytest.mark.parametrize("n,pml,vti,src", [
    ((36, 50, 54), 7, True, 0),    # nz % 4 == 2, ny % 4 == 2, radix 9 x 6
    ((42, 54, 98), 9, False, 1),   # radix 14 x 7, isotropic, explosive
    ((40, 42, 162), 5, True, 1),   # three stages 9 6 3
    ((54, 40, 64), 7, True, 0),    # 8 x 8: shuffles over 8 lanes
    ((50, 36, 128), 9, False, 0),  # 16 x 8
    ((36, 48, 150), 11, True, 0),  # 15 x 10
    ((250, 36, 40), 5, False, 0),  # x in three stages 10 5 5
    ((36, 216, 48), 7, True, 0),   # y in three stages 6 6 6
])
def test_against_oracle(qvti, oracle, n, pml, vti, src):
    c = _case(n, pml, seed=sum(n))
    ours = qvti.run_case(c, vti=vti, src_type=src, ref_offset=False, want_state=True)
    ref = oracle.run_case(c, vti=vti, src_type=src, ref_offset=False, want_state=True)
    for f, name in enumerate(qvti.FIELDS):
        e = qc.relL2(ours["state"][f], ref["state"][f])
        assert e <= TOL, "%s %s relL2 %.3g" % (n, name, e)


def test_compiled_and_runtime_velocity_kernels_agree(qvti):
    """k_dv against the runtime kernels on the same shot: FP32 rounding."""
    c = _case((64, 40, 64), 6, 3)
    a = qvti.run_case(c, vti=True, want_state=True)
    b = qvti.run_case(c, vti=True, tiles=[16, 16, 0, 0, 0, 0], want_state=True)
    for i in range(9):
        # the tile tests' rounding bound
        assert qc.relL2(a["state"][i], b["state"][i]) <= 2e-5
