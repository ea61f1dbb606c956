"""Records and images that are nothing but the transforms' rounding.

    python tests/golden/make_rounding.py OUT.npz [LIBQVTI.SO]      (on a B200)

A global transform spreads its rounding over the whole grid, so a receiver that
the wave has not reached records the last bits of every transform since the
first step.  Two evaluations of the scheme that round one product differently
agree to 1e-6 in the wavefield and to 1e-4 in such a record, and the shots of one
survey are compared with one another and with those of an earlier run: the
library keeps the rounding of its step from one form of its kernels to the next.
The fixture holds what the library of commit 657271f gave (CUDA 12.9), whose step
kernels were scalar.
"""
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
import qvti_cases as qc  # noqa: E402

# grid, C-PML, VTI, source type, steps.  z lengths of one and of two radices per
# stage, of three stages, odd radices, and runtime lengths; the source lies as
# deep below the receivers as the grid allows
SHOTS = {
    "z96": ((64, 48, 96), 6, True, 0, 24),
    "z120": ((54, 60, 120), 7, False, 1, 24),
    "z128": ((96, 42, 128), 6, True, 0, 20),
    "z98": ((40, 84, 98), 5, True, 1, 24),
    "z162": ((36, 50, 162), 6, False, 0, 16),
    "z256": ((72, 64, 256), 6, True, 0, 12),
    "z32": ((32, 32, 32), 4, True, 0, 16),
    "z56": ((70, 128, 56), 6, False, 0, 20),
    "x320": ((320, 40, 48), 5, True, 0, 12),
    "y360": ((48, 360, 64), 5, True, 0, 12),
}
TC = {"tc256": ((48, 256, 64), 5, True, 0, 12)}  # the tensor-core form of the y transforms
RTM = {"rtm64": ((64, 80, 72), 10, 40, 4)}  # grid, C-PML, steps, media


def case(n, pml, nt):
    """Layers with cell-wise integer perturbations: the same on every machine."""
    rng = np.random.default_rng(sum(n))
    vp = (2200 + 60 * (np.arange(n[2]) // 12) % 700)[None, None, :] + rng.integers(-60, 61, n)
    vp = vp.astype(np.float32)
    q = (40 + rng.integers(0, 100, n)).astype(np.float64)
    rx = np.arange(pml, n[0] - pml, 3, dtype=np.int32)
    c = dict(name="rounding", ntx=n[0], nty=n[1], ntz=n[2], pml=pml, nt=nt, dx=10.0, dy=11.0, dz=9.0, dt=0.6e-3,
             f0=30.0, velp=vp, vels=(vp * np.float32(0.5625)), rho=(vp * np.float32(0.875)),
             gama_p=qc.gamma_of_q(q), gama_s=qc.gamma_of_q(0.5 * q), rik=qc.ricker(nt, 0.6e-3, 60.0),
             s_ix=n[0] // 2, s_iy=n[1] // 2, s_iz=n[2] - pml - 2, r_iz=pml + 1, r_ix=rx,
             r_iy=np.full(rx.size, n[1] // 2, np.int32), rnx_max=rx.size, rny_max=1)
    c["eps"] = (rng.integers(0, 26, n) / np.float32(128)).astype(np.float32)
    c["delta"] = (rng.integers(0, 13, n) / np.float32(128)).astype(np.float32)
    return c


def shot(qvti, name):
    n, pml, vti, src, nt = {**SHOTS, **TC}[name]
    return np.asarray(qvti.run_case(case(n, pml, nt), vti=vti, src_type=src, ref_offset=False,
                                    form=qvti.FORM_TC if name in TC else qvti.FORM_PLAIN)["rec"], np.float32)


def rtm(qvti, name):
    """Both images on the plane of the receivers' line."""
    n, pml, nt, media = RTM[name]
    c = case(n, pml, nt)
    t = np.arange(nt, dtype=np.int64)[:, None]
    x = np.arange(c["r_ix"].size, dtype=np.int64)[None, :]
    obs = np.stack([(((t - 12) * (17 + k) + x * 5) % 23 - 11).astype(np.float32) for k in range(3)])
    im = qvti.rtm_shot(c, obs, media=media, snap_every=5, illum_eps=1e-2, ref_offset=False)
    return np.stack([a[:, n[1] // 2, :] for a in im])


if __name__ == "__main__":
    import importlib.util
    spec = importlib.util.spec_from_file_location(
        "qvti_b200", os.path.join(os.path.dirname(os.path.dirname(HERE)), "q-vti_b200", "qvti.py"))
    qvti = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(qvti)
    if len(sys.argv) > 2:
        qvti.LIB_PATH = sys.argv[2]
    out = {k: shot(qvti, k) for k in {**SHOTS, **TC}}
    out.update({k: rtm(qvti, k) for k in RTM})
    np.savez_compressed(sys.argv[1], **out)
    for k, v in out.items():
        print(k, v.shape, float(np.abs(v).max()))
