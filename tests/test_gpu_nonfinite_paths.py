"""A non-finite cell is seen by every kernel that steps packed lattices and batches:
the staged one, and the one of a thread per cell at both kinds of width."""
import numpy as np
import pytest

from fixtures import packed_planes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _inject_nan(lat):
    """NaN into f_0 of one fluid cell of the packed state (FP32 storage), on the host."""
    ys, xs = np.nonzero(~lat.geometry.solid[:, lat.W // 4:3 * lat.W // 4])
    y, x = int(ys[len(ys) // 2]), int(xs[len(xs) // 2]) + lat.W // 4
    lat.ppop[lat.pcur][4 * (y * lat.W + x):4 * (y * lat.W + x) + 4].view(torch.float32).fill_(float("nan"))


@pytest.mark.parametrize("W,rows", [(128, 16), (128, 0), (92, 0)], ids=["staged", "tile", "tile_odd_width"])
def test_a_single_lattice_reports_it(W, rows):
    from fingering_dynamics_gb300 import geometry as geo
    from fingering_dynamics_gb300.lattice import Lattice
    from fingering_dynamics_gb300.params import walls_reference_params
    prm = walls_reference_params().with_size(48, W)
    g = geo.build_geometry(48, W, rects=[((40, 12), (46, 20))], walls=True)
    ok, bad = Lattice(prm, g, dtype="f32"), Lattice(prm, g, dtype="f32")
    ok.enter_fused()
    ok.check_finite()  # clear
    ok.advance(4, rows_per_warp=rows)
    ok.check_finite()
    bad.enter_fused()
    _inject_nan(bad)
    bad.advance(2, rows_per_warp=rows)
    with pytest.raises(FloatingPointError):
        bad.check_finite()
    ok.check_finite()  # cleared by the raising call


@pytest.mark.parametrize("rows,kernel", [(16, "staged"), (32, "tile")])
def test_a_batch_quarantines_the_member(rows, kernel):
    """The flagged member is not stepped any more and leaves the next table, the
    others go on as alone, and a cleared flag takes it back."""
    from fingering_dynamics_gb300.ensemble import Ensemble, ensemble_specs
    from fingering_dynamics_gb300.lattice import Lattice
    members = [s.build() for s in ensemble_specs(4, seed=3, sizes_w=(64, 128, 256), sizes_h=(48, 64, 96), ratio=(2.0, 5.0))]
    ens = Ensemble(members, dtype="f32", rows_per_strip=rows)
    solo = [Lattice(m[0], m[1], dtype="f32") for m in members]
    for lat in solo:
        lat.enter_fused()
    assert ens.kernel == kernel
    bad = ens.lattices[2]

    def go(n):
        ens.step(n)
        torch.cuda.synchronize()
        for k in (0, 1, 3):
            solo[k].advance(n)
            got, ref = ens.lattices[k], solo[k]
            assert torch.equal(packed_planes(got.ppop[got.pcur], got.H, got.W, "f32"),
                               packed_planes(ref.ppop[ref.pcur], ref.H, ref.W, "f32")), k
            assert torch.equal(got.side[got.scur], ref.side[ref.scur]), k

    go(4)
    assert ens.member_status() == [False] * 4
    good = [b.clone() for b in bad.ppop], [s.clone() for s in bad.side]
    _inject_nan(bad)
    go(3)
    assert ens.member_status() == [False, False, True, False]
    frozen = [b.clone() for b in bad.ppop]
    go(6)
    full = ens.tiles
    ens.configure(*ens.config)  # a table without the member
    assert ens.tiles < full and ens.kernel == kernel
    go(5)
    assert all(torch.equal(a, b) for a, b in zip(frozen, bad.ppop)), "a quarantined member was stepped"
    # restored (an even number of iterations on, so in the same buffer), cleared and configured again it steps on
    for to, of in zip(bad.ppop + bad.side, good[0] + good[1]):
        to.copy_(of)
    assert ens.member_status(clear=True)[2]
    ens.configure(*ens.config)
    assert ens.tiles == full and ens.member_status() == [False] * 4
    solo[2].advance(4)
    ens.step(4)
    solo[2].advance(4)
    torch.cuda.synchronize()
    assert ens.member_status() == [False] * 4
    assert torch.equal(packed_planes(bad.ppop[bad.pcur], bad.H, bad.W, "f32"),
                       packed_planes(solo[2].ppop[solo[2].pcur], bad.H, bad.W, "f32"))
    ens.close()
