"""Paths of the fused step that ordinary runs do not take: the FP64 cell that gives up
after it has stored some directions, the tile kernel's 64-bit offsets, and its
arithmetic at widths that are not a multiple of 8 with scaled storage."""
import ctypes as C

import numpy as np
import pytest

from oracle.lbm_oracle import OracleParams, OracleState, bottom_top_wall, halfway_bounceback_rec, stream

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _params(H, W, variant):
    from fingering_dynamics_gb300.params import periodic_reference_params, walls_reference_params
    prm = (walls_reference_params if variant == "walls" else periodic_reference_params)().with_size(H, W)
    if variant == "walls":
        prm.M, prm.u0, prm.inlet_ux = 3.0, 0.006, np.full(H, 0.006)
    return prm


def _oracle_after(lat, f, g):
    """The oracle's state one iteration on: `lat` (reference mode) holds the fields, f and g are its populations
    after the collision; streams, applies the boundaries, updates the fields and collides."""
    prm, geo = lat.params, lat.geometry
    op = OracleParams(H=prm.H, W=prm.W, variant=prm.variant, tau=prm.tau, eta_n=prm.eta_n, M=prm.M, a=prm.a,
                      kappa=prm.kappa, gamma=prm.gamma, psi_wall=prm.psi_wall, inlet_ux=prm.inlet_ux,
                      outlet_coef=prm.outlet_coef)
    st = OracleState(op, geo.solid, lat.psi.double().cpu().numpy())
    st.np2 = lat.np2.double().cpu().numpy()
    st.f, st.g = stream(f), stream(g)
    if geo.corner_list:
        halfway_bounceback_rec(geo.corner_list, f, g, st.f, st.g)
    if prm.variant == "walls":
        bottom_top_wall(f[:, 1:-1], g[:, 1:-1], st.f[:, 1:-1], st.g[:, 1:-1])
    st.zou_he()
    st.macros()
    st.collide()
    return st


@pytest.mark.parametrize("H,W", [(40, 64), (512, 520)])  # tiles of 4 rows, of 8 rows
def test_fp64_cell_that_gives_up_halfway(H, W):
    """A g of 1e-130 (outside the fast arithmetic's range, but a number) in each
    direction, so that the cell stops after the directions before it were stored;
    also in cells of the inlet and of the outlet column."""
    from fingering_dynamics_gb300 import geometry as geo
    from fingering_dynamics_gb300.lattice import Lattice
    lat = Lattice(_params(H, W, "periodic"), geo.build_geometry(H, W), dtype="f64")
    lat.step(3)
    keep = Lattice(lat.params, lat.geometry, dtype="f64")
    keep.psi.copy_(lat.psi)
    keep.np2.copy_(lat.np2)
    lat.enter_fused()
    pop = lat.pop[lat.cur]
    for i in range(9):
        pop[9 + i, 4 * i + 1, 6 * i + 4] = 1e-130
    pop[9 + 3, 7, 1] = 1e-130       # arrives in the inlet column
    pop[9 + 1, 9, W - 2] = 1e-130   # and in the outlet column
    st = _oracle_after(keep, pop[:9].cpu().numpy(), pop[9:].cpu().numpy())
    lat.advance(1)
    assert torch.equal(lat.f.cpu(), torch.from_numpy(st.f)) and torch.equal(lat.g.cpu(), torch.from_numpy(st.g))


def test_tile_step_with_64_bit_offsets():
    """Planes above 4 GB: a lattice of 12 columns that repeats 30 rows steps as
    those 30 rows do (the periodic variant wraps in y)."""
    from fingering_dynamics_gb300 import _lib as L
    from fingering_dynamics_gb300 import geometry as geo
    from fingering_dynamics_gb300.lattice import Lattice, _ptr
    h, W, k = 30, 12, 331500
    H = h * k
    assert 9 * H * W * 4 >= 1 << 32
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB")
    lat = Lattice(_params(h, W, "periodic"), geo.build_geometry(h, W, rects=[((4, 8), (7, 12))]), dtype="f32")
    lat.step(3)
    lat.enter_fused()
    lat.advance(2)
    planes = torch.empty((18, h, W), device="cuda")
    small, big = L.fd_params.from_buffer_copy(lat.prm), L.fd_params.from_buffer_copy(lat.prm)
    big.H = H
    st = C.byref(lat.storage)
    L.call("fd_unpack", C.byref(small), st, _ptr(lat.current_buffer()), L.FD_F32, _ptr(planes), None)

    def stepped(prm, times):
        rows = lambda t: t.repeat(*([1] * (t.dim() - 1)), times).contiguous()  # noqa: E731
        mask = rows(lat.mask.reshape(-1))
        inlet, side = rows(lat.inlet_ux), rows(lat.side[lat.scur])
        other = torch.empty_like(side)
        ref = planes.reshape(18, 1, -1).expand(18, times, h * W).clone(memory_format=torch.contiguous_format)
        pop = [torch.empty(L.lib().fd_packed_bytes(h * times, W, st), dtype=torch.uint8, device="cuda") for _ in range(2)]
        L.call("fd_pack", C.byref(prm), L.FD_F32, _ptr(ref), st, _ptr(pop[0]), None)
        L.call("fd_fused_step_packed", C.byref(prm), st, _ptr(mask), _ptr(inlet), _ptr(pop[0]), _ptr(pop[1]), _ptr(side),
               _ptr(other), 3, 0, None)
        L.call("fd_unpack", C.byref(prm), st, _ptr(pop[1]), L.FD_F32, _ptr(ref), None)
        return ref, other.view(6, times, h)

    want, want_side = stepped(small, 1)
    got, got_side = stepped(big, k)
    assert not torch.equal(want.view_as(planes), planes)
    for p in range(18):
        assert bool((got[p] == want[p]).all()), p
    assert bool((got_side == want_side).all())


@pytest.mark.parametrize("dtype,rounding,scales", [("f32", "nearest", (0, 0)), ("f16", "stochastic", (0, 0)),
                                                   ("f16", "nearest", (4, 2)), ("f16", "stochastic", (5, 1)),
                                                   ("bf16", "stochastic", (3, 0)), ("bf16", "nearest", (0, 4))])
@pytest.mark.parametrize("H,W,variant", [(3, 4, "walls"), (6, 12, "periodic"), (16, 36, "walls"), (34, 100, "periodic"),
                                         (33, 100, "walls")])
def test_odd_widths_follow_the_oracle(H, W, variant, dtype, rounding, scales):
    """One step at a width that is not a multiple of 8, from a known packed state, in
    64 bits.  A stored value v (f as its deviation) may be off by its rounding,
    u |v| (half an ulp to nearest, an ulp stochastically), by half a subnormal step of
    FP16, and by 128 roundings of FP32 arithmetic on values up to 1."""
    from fingering_dynamics_gb300 import _lib as L
    from fingering_dynamics_gb300 import geometry as geo
    from fingering_dynamics_gb300.lattice import Lattice, _ptr
    rects = [((W // 2, H // 2 - 1), (W // 2 + 2, H // 2 + 1))] if H >= 16 else []
    g = geo.build_geometry(H, W, rects=rects, walls=variant == "walls")
    rho0 = 1 + 1e-3 * np.random.default_rng(H + W).standard_normal((H, W))
    lat = Lattice(_params(H, W, variant), g, dtype=dtype, rounding=rounding, seed=11, rho0=rho0)
    lat.storage.f_scale_log2, lat.storage.g_scale_log2 = scales
    lat.step_reference(3)
    keep = Lattice(lat.params, g, dtype=dtype)
    keep.psi.copy_(lat.psi)
    keep.np2.copy_(lat.np2)

    def planes():
        out = torch.empty((18, H, W), dtype=torch.float64, device="cuda")
        L.call("fd_unpack", C.byref(lat.prm), C.byref(lat.storage), _ptr(lat.current_buffer()), L.FD_F64, _ptr(out), None)
        return out.cpu().numpy()
    lat.enter_fused()
    before = planes()
    st = _oracle_after(keep, before[:9], before[9:])
    lat.advance(1)
    after = planes()
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)[:, None, None]
    ulp = {"f32": 2.0 ** -23, "f16": 2.0 ** -10, "bf16": 2.0 ** -7}[dtype] * (1.0 if rounding == "stochastic" else 0.5)
    for got, want, scale in ((after[:9] - w, st.f - w, scales[0]), (after[9:], st.g, scales[1])):
        assert np.isfinite(got).all()
        tol = ulp * np.abs(want) + 128 * 2.0 ** -24 + (2.0 ** -24 / 2.0 ** scale if dtype == "f16" else 0.0)
        assert (np.abs(got - want) <= tol).all(), np.abs(got - want).max()
