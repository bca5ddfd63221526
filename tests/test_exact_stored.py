"""The per-function FP64 collision's cell arithmetic (exact_stored and exact_collide of
csrc/fd_exact_cell.h), compiled for the host, against the oracle's operand order: stored
fields are taken in the ranges that the fused step takes, with the same bits, and
refused outside."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle.lbm_oracle import W9, OracleParams, OracleState

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "fd_exact_cell.h"
using namespace fd;
extern "C" void cells(const double* c, long n, const double* m, double* f, double* g, unsigned char* ok) {
  const ExactConst k = make_exact_const(c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9], c[10]);
  for (long j = 0; j < n; ++j) {
    double v[9], fc[9], fo[9], go[9];
    for (int i = 0; i < 9; ++i) { v[i] = m[i * n + j]; fc[i] = f[i * n + j]; }
    ok[j] = exact_collide(k, exact_stored(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8]), fc,
                          [&](int i) { return g[i * n + j]; }, [&](int i, double a, double b) { fo[i] = a; go[i] = b; });
    if (ok[j]) for (int i = 0; i < 9; ++i) { f[i * n + j] = fo[i]; g[i * n + j] = go[i]; }
  }
}
"""


@pytest.fixture(scope="module")
def cells(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("exact_stored")
    (d / "cell.cpp").write_text(SRC)
    lib = str(d / "cell.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                    os.path.join(REPO, "fingering_dynamics_gb300", "csrc"), str(d / "cell.cpp"), "-o", lib], check=True)
    return C.CDLL(lib).cells


def collide(cells, st):
    """(f, g, taken) of every cell of an oracle state whose fields are its stored ones."""
    p = st.prm
    ca0 = 3.0 * (1.0 - W9[0])
    const = np.array([W9[0], W9[1], p.a, p.kappa, p.eta_n, p.eta_n * p.M, ca0, ca0 * p.gamma, 3 * p.gamma, 1 / 3,
                      1.0 / p.tau])
    m = np.ascontiguousarray(np.stack([v.reshape(-1) for v in (st.rho, st.ux, st.uy, st.p, st.mu, st.mix_tau, st.psi, st.npx,
                                                               st.npy)]))
    f, g = (np.ascontiguousarray(v.reshape(9, -1)).copy() for v in (st.f, st.g))
    n = m.shape[1]
    ok = np.zeros(n, np.uint8)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    with np.errstate(all="ignore"):
        cells(ptr(const), C.c_long(n), ptr(m), ptr(f), ptr(g), ptr(ok))
    return f, g, ok.astype(bool)


def state(scale):
    """psi, g and p of every second cell scaled down by `scale`."""
    H, W = 16, 64
    rng = np.random.default_rng(3)
    prm = OracleParams(H=H, W=W, variant="periodic", tau=0.789, eta_n=1 / 30, M=4.0, a=-0.0125, kappa=0.0125, gamma=7.0,
                       psi_wall=-0.5, inlet_ux=np.zeros(H), outlet_coef=2 / 3)
    st = OracleState(prm, np.zeros((H, W), bool), np.tanh(rng.normal(0, 1, (H, W))))
    st.f = W9[:, None, None] * (1 + rng.normal(0, 1e-3, (9, H, W)))
    st.macros()
    st.psi[:, ::2] *= scale
    st.g[:, :, ::2] *= scale
    st.p = st.p.reshape(H, W)
    st.p[:, ::2] *= scale
    st.p = st.p.reshape(-1)
    return st


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -60, 2.0 ** -130, 2.0 ** -390, 0.0])
def test_small_stored_fields_are_taken(cells, scale):
    st = state(scale)
    f, g, ok = collide(cells, st)
    assert ok.all()
    st.collide()
    assert np.array_equal(f, st.f.reshape(9, -1)) and np.array_equal(g, st.g.reshape(9, -1))


@pytest.mark.parametrize("field,value", [("psi", 2.0 ** -401), ("psi", np.nan), ("psi", np.inf), ("p", 2.0 ** 801), ("p", -np.inf),
                                         ("npx", 2.0 ** -801), ("npy", np.nan), ("rho", 2.0 ** 101), ("ux", 2.0 ** 401),
                                         ("uy", np.inf), ("mu", 2.0 ** -801), ("mix_tau", 0.0), ("mix_tau", np.nan)])
def test_stored_fields_out_of_range_are_refused(cells, field, value):
    st = state(1.0)
    getattr(st, field).reshape(-1)[100] = value
    f, g, ok = collide(cells, st)
    assert np.flatnonzero(~ok).tolist() == [100]
    assert np.array_equal(f[:, 100], st.f.reshape(9, -1)[:, 100]) and np.array_equal(g[:, 100], st.g.reshape(9, -1)[:, 100])
