"""F*(U-, U+, n) - F(U-).n of the HLLC flux as the resident barotropic form computes it (flux.cuh,
compiled for the host here) against the oracle's HLLC, over its branches."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import pyoracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
G, DRY = 9.81, 1e-10
NORMAL = np.array([[-1.0, 0.0], [1.0, 0.0], [0.0, -1.0], [0.0, 1.0]])


@pytest.fixture(scope="module")
def diff(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    so = str(tmp_path_factory.mktemp("flux") / "flux_diff.so")
    subprocess.run(["g++", "-std=c++20", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "drifter_b200", "csrc"), "-I", CUDA,
                    os.path.join(ROOT, "tests", "cpp", "flux_diff.cpp"), "-o", so],
                   check=True, capture_output=True, text=True)
    fn = C.CDLL(so).hllc_diff_batch

    def call(UL, UR, side):
        d = np.empty_like(UL)
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        fn(len(UL), p(UL), p(UR), p(side), C.c_double(G), p(d))
        return d

    return call


def _states(kind, rng, n):
    """Depths and outward and tangential velocities of the two sides, (n, 2) each."""
    h = rng.uniform(0.5, 3.0, (n, 2))
    un, ut = rng.normal(0, 1, (n, 2)), rng.normal(0, 1, (n, 2))
    c = np.sqrt(G * h.max(1, keepdims=True))
    if kind == "out":
        un = rng.uniform(1.2, 4.0, (n, 2)) * c
    elif kind == "in":
        un = -rng.uniform(1.2, 4.0, (n, 2)) * c
    elif kind == "transcritical":
        un = rng.uniform(-2.0, 2.0, (n, 2)) * c
    elif kind == "depths":
        h = 10.0 ** rng.uniform(-3, 3, (n, 2))
    dry = rng.choice([0.0, 1e-12, 5e-11, -1e-12, -1e-3], (n, 2))
    if kind in ("dry_in", "dry_both"):
        h[:, 0] = dry[:, 0]
    if kind in ("dry_out", "dry_both"):
        h[:, 1] = dry[:, 1]
    if kind.startswith("dry"):
        un, ut = 0.1 * un, 0.1 * ut
    return h, un, ut


@pytest.mark.parametrize("kind", ["subcritical", "out", "in", "transcritical", "depths", "dry_in", "dry_out", "dry_both"])
def test_hllc_face_difference_matches_oracle(diff, kind):
    """Tolerance 1e-12 of h (|u| + c) and h (|u| + c)^2, the largest of the two sides': some 50 rounded
    operations, amplified at most by (1 + |u| / c)^2 = 25 for these states, against the oracle's F* and
    F(U-), whose difference rounds at 1e-16 of the same scale."""
    rng = np.random.default_rng(sum(map(ord, kind)))
    n = 1200
    h, un, ut = _states(kind, rng, n)
    side = (np.arange(n) % 4).astype(np.int32)
    nr = NORMAL[side]
    tan = np.stack([-nr[:, 1], nr[:, 0]], 1)
    hw = np.maximum(h, DRY)  # momenta of the clamped depth
    U = [np.ascontiguousarray(np.column_stack([h[:, k], hw[:, k, None] * (un[:, k, None] * nr + ut[:, k, None] * tan)]))
         for k in (0, 1)]
    d = diff(U[0], U[1], side)
    ref = np.array([O.sw_flux("hllc", U[0][i], U[1][i], nr[i, 0], nr[i, 1]) for i in range(n)])
    u = U[0][:, 1:] / hw[:, :1]
    Fm = np.column_stack([hw[:, 0] * un[:, 0], hw[:, :1] * u * un[:, :1] + 0.5 * G * hw[:, :1] ** 2 * nr])
    # which branches the states take
    c = np.sqrt(G * hw)
    SL, SR = (un - c).min(1), (un + c).max(1)
    den = hw[:, 0] * (SL - un[:, 0]) - hw[:, 1] * (SR - un[:, 1])
    out, inn = SL >= 0, SR <= 0
    if kind == "out":
        assert out.all()
    elif kind == "in":
        assert inn.all()
    elif kind == "dry_both":
        assert (np.abs(den) <= 1e-10).all()
    else:
        assert (~out & ~inn).sum() > 100
    v = (np.hypot(un, ut) + c).max(1)
    scale = hw.max(1)[:, None] * np.column_stack([v, v * v, v * v])
    err = np.abs(d - (ref - Fm)) / scale
    assert np.isfinite(d).all() and err.max() <= 1e-12, (err.max(), err.argmax())
