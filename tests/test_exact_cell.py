"""The FP64 step's cell arithmetic (csrc/fd_exact_cell.h), compiled for the
host, against the oracle's operand order: every bit of the macroscopic fields'
collision must agree, and values outside its range must be refused."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle.lbm_oracle import W9, OracleParams, OracleState, _nbrs, _padded_psi

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "fd_exact_cell.h"
using namespace fd;
extern "C" void cells(const double* c, long n, const double* nb, double* f, double* g, unsigned char* ok) {
  const ExactConst k = make_exact_const(c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9], c[10]);
  for (long j = 0; j < n; ++j) {
    double v[9], fc[9], fo[9], go[9];
    for (int i = 0; i < 9; ++i) { v[i] = nb[i * n + j]; fc[i] = f[i * n + j]; }
    const ExactStencil s = exact_stencil(k, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8]);
    ok[j] = exact_cell(k, v[0], s, fc, [&](int i) { return g[i * n + j]; },
                       [&](int i, double a, double b) { fo[i] = a; go[i] = b; });
    if (ok[j]) for (int i = 0; i < 9; ++i) { f[i * n + j] = fo[i]; g[i * n + j] = go[i]; }
  }
}
"""


@pytest.fixture(scope="module", params=[0, 58])  # products in integer arithmetic: none, all
def cells(tmp_path_factory, request):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("exact_cell")
    (d / "cell.cpp").write_text(SRC)
    lib = str(d / "cell.so")
    subprocess.run([cxx, "-O2", f"-DFD_EXACT_INT_PRODUCTS={request.param}", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                    os.path.join(REPO, "fingering_dynamics_gb300", "csrc"), str(d / "cell.cpp"), "-o", lib], check=True)
    return C.CDLL(lib).cells


def oracle_state(H, W, seed, spread, eta=(1 / 30, 4.0)):
    rng = np.random.default_rng(seed)
    prm = OracleParams(H=H, W=W, variant="periodic", tau=0.789, eta_n=eta[0], M=eta[1], a=-0.0125, kappa=0.0125,
                       gamma=7.0, psi_wall=-0.5, inlet_ux=np.zeros(H), outlet_coef=2 / 3)
    psi = np.tanh(np.cumsum(rng.normal(0, 0.3, (H, W)), axis=1)).round(rng.integers(1, 4))
    st = OracleState(prm, np.zeros((H, W), bool), psi)
    st.f = W9[:, None, None] * (1 + rng.normal(0, spread, (9, H, W)))
    st.g = st.g + rng.normal(0, spread * 0.1, (9, H, W)) * (rng.random((H, W)) < 0.7)
    st.macros()
    return st


def run(cells, st, f, g):
    p = st.prm
    ca0 = 3.0 * (1.0 - W9[0])
    const = np.array([W9[0], W9[1], p.a, p.kappa, p.eta_n, p.eta_n * p.M, ca0, ca0 * p.gamma, 3 * p.gamma, 1 / 3,
                      1.0 / p.tau])
    nb = np.ascontiguousarray(np.stack([v.reshape(-1) for v in _nbrs(_padded_psi(st.psi, st.solid, p))]))
    n = nb.shape[1]
    ok = np.zeros(n, np.uint8)
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    with np.errstate(all="ignore"):
        cells(ptr(const), C.c_long(n), ptr(nb), ptr(f), ptr(g), ptr(ok))
    return ok.astype(bool)


@pytest.mark.parametrize("spread", [0.0, 1e-9, 1e-3, 0.1])
@pytest.mark.parametrize("eta", [(1 / 30, 4.0), (0.0963, 20.0), (1 / 30, 1.0)])
def test_cell_equals_the_reference_order(cells, spread, eta):
    st = oracle_state(96, 512, int(1e6 * spread) + int(eta[1]), spread, eta)
    f, g = (np.ascontiguousarray(v.reshape(9, -1)).copy() for v in (st.f, st.g))
    ok = run(cells, st, f, g)
    assert ok.all()
    st.collide()
    assert np.array_equal(f, st.f.reshape(9, -1))
    assert np.array_equal(g, st.g.reshape(9, -1))


def test_rounding_noise_is_in_range(cells):
    """Far from the interface u and g are products of rounding errors (1e-36 and
    below): such cells are taken, with the same bits."""
    H, W = 8, 160
    prm = OracleParams(H=H, W=W, variant="periodic", tau=0.789, eta_n=1 / 30, M=4.0, a=-0.0125, kappa=0.0125, gamma=7.0,
                       psi_wall=-0.5, inlet_ux=np.full(H, 0.003), outlet_coef=2 / 3)
    st = OracleState(prm, np.zeros((H, W), bool), np.where(np.arange(W) < 20, 1.0, -1.0) * np.ones((H, 1)))
    small = 0
    for _ in range(40):
        st.step()
        f, g = (np.ascontiguousarray(v.reshape(9, -1)).copy() for v in (st.f, st.g))
        small += int(((st.g != 0) & (abs(st.g) < 2.0 ** -100)).sum() + ((st.uy != 0) & (abs(st.uy) < 2.0 ** -100)).sum())
        assert run(cells, st, f, g).all()
        want = OracleState(prm, st.solid, st.psi.copy())
        want.f, want.g = st.f.copy(), st.g.copy()
        want.macros()
        want.collide()
        assert np.array_equal(f, want.f.reshape(9, -1)) and np.array_equal(g, want.g.reshape(9, -1))
    assert small > 0


def test_values_out_of_range_are_refused_untouched(cells):
    st = oracle_state(8, 64, 5, 1e-3)
    f, g = (np.ascontiguousarray(v.reshape(9, -1)).copy() for v in (st.f, st.g))
    bad = [np.inf, -np.inf, np.nan, 1e300, -1e-290]
    for j, v in enumerate(bad):
        f[:, 3 * j + 1] = 0.0
        f[2, 3 * j + 1] = v
    st.psi[5, 40] = np.nan
    keep = f.copy(), g.copy()
    ok = run(cells, st, f, g)
    refused = np.flatnonzero(~ok)
    assert set(3 * j + 1 for j in range(len(bad))) <= set(refused)
    assert 5 * 64 + 40 in refused and 5 * 64 + 41 in refused  # its own cell and the neighbours whose stencils read it
    assert np.array_equal(f[:, refused], keep[0][:, refused], equal_nan=True)
    assert np.array_equal(g[:, refused], keep[1][:, refused], equal_nan=True)
