"""Tiles, ring and shared-memory windows of the persistent tcgen05 convolutions
(csrc/sg_conv.cu, csrc/sg_conv_plan.h), no GPU.

The plan is compiled for the host.  A stage's shared memory is rebuilt as its swizzled
tensor-map box fills it (NaN elsewhere), every tap's operand is read through the window
the kernel's descriptors give it (row m at start + m pixels, the swizzle a function of
the address), and the sums of the pixels that the epilogue keeps are compared with a
direct convolution."""
import os
import shutil
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "sg_conv_plan.h"
int main(int argc, char** argv) {
  int a[5];
  for (char line[256]; std::fgets(line, sizeof line, stdin);) {
    if (line[0] == 't') {
      std::sscanf(line + 1, "%d %d %d", a, a + 1, a + 2);
      int bw = 0, rows = 0;
      sg::tile_box(a[0], a[1], a[2], bw, rows);
      std::printf("%d %d\n", bw, rows);
    } else {
      std::sscanf(line + 1, "%d %d %d %d %d", a, a + 1, a + 2, a + 3, a + 4);
      const sg::ConvRing r = sg::conv_ring(a[0], a[1], a[2], a[3], a[4]);
      std::printf("%d %d\n", r.resident, r.stages);
    }
  }
  return 0;
}
"""
BM, S_MAX = 128, 6


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("conv_plan")
    (d / "p.cpp").write_text(DRIVER)
    exe = str(d / "p")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(REPO, "fingering_dynamics_gb300", "csrc"), "-o", exe,
                    str(d / "p.cpp")], check=True)

    def ask(kind, rows):
        text = "".join(f"{kind} {' '.join(map(str, r))}\n" for r in rows)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()
        return [tuple(map(int, out[k:k + 2])) for k in range(0, len(out), 2)]
    return ask


def cfg(BN, R, CH):
    """CvCfg<BN, R, CH, .>"""
    row = 2 * CH
    up = lambda v: (v + 1023) // 1024 * 1024  # noqa: E731
    a_tx = (R + 2) * 130 * row
    return {"ROW": row, "A_TX": a_tx, "A": up(a_tx), "TAP": BN * row, "B": up(9 * BN * row),
            "TAIL": (2 * S_MAX + 5) * 8 + BN * 4 + 16 + 1024}


@pytest.mark.parametrize("gap", [0, 2])
def test_tiles_of_every_width(plan, gap):
    """gap 0: k_conv3x3_narrow, a box per tap; gap 2: the FLAT form, one halo box."""
    shapes = [(H, W, gap) for W in range(1, 2600) if W % 128 for H in (1, 2, 3, 50, 257)]
    for (H, W, _), (bw, rows) in zip(shapes, plan("t", shapes)):
        pitch = bw + gap
        assert 1 <= bw <= min(W, BM) and rows >= 1 and -(-W // bw) * bw >= W
        assert (rows - 1) * pitch + bw <= BM                 # the tile's pixels among the operand rows
        assert pitch <= 256 and rows + 2 <= 256              # tensor-map boxes
        for CH in (16, 32):
            c = cfg(16, 1, CH)
            if gap:
                assert (rows + 2) * pitch * c["ROW"] <= c["A_TX"]
                assert (2 * pitch + 2 + BM) * c["ROW"] <= c["A"]       # the last tap's window, rows past the tile too
                assert (rows + 1) * pitch + bw + 2 <= (rows + 2) * pitch  # and what is kept of it lies in the box


@pytest.mark.parametrize("BN,R,CH", [(BN, R, CH) for BN in (16, 32, 64, 96, 128) for R in (1, 2, 4) for CH in (16, 32)
                                     if 2 * R * BN <= 512])
def test_ring_fits(plan, BN, R, CH):
    c = cfg(BN, R, CH)
    room = 227 * 1024 - c["TAIL"]
    asked = [(nk, c["A"], c["B"], room, S_MAX) for nk in range(1, 65)]
    for (nk, a, b, _, _), (resident, stages) in zip(asked, plan("r", asked)):
        assert 1 <= stages <= S_MAX and (stages >= 2 or nk == 1 or not resident)
        used = stages * (a + (0 if resident else b)) + (nk * b if resident else 0)
        assert used % 1024 == 0 and used <= room
        assert resident or nk * b + 2 * a > room or nk == 1


def swizzle(addr, row):
    """The 16-byte unit of an address in a pattern of rows of 32, 64 or 128 bytes."""
    bits = {32: 1, 64: 3, 128: 7}[row]
    return addr ^ (((addr >> 7) & bits) << 4)


def stage(x, n, x0, y0, box_w, box_h, ch0, CH, size):
    """A stage as the box (CH channels, box_w pixels, box_h rows) from (ch0, x0, y0, n) fills it, per element."""
    st = np.full(size // 2, np.nan)
    N, H, W, _ = x.shape
    for p in range(box_w * box_h):
        yy, xx = y0 + p // box_w, x0 + p % box_w
        v = x[n, yy, xx, ch0:ch0 + CH] if 0 <= yy < H and 0 <= xx < W else np.zeros(CH)
        for u in range(CH // 8):
            o = swizzle(p * 2 * CH + 16 * u, 2 * CH) // 2
            st[o:o + 8] = v[8 * u:8 * u + 8]
    return st


def window(st, start, CH, s):
    """128 operand rows x 16 channels (slice s of the chunk) of the window that starts `start` pixels in."""
    out = np.empty((BM, 16))
    for m in range(BM):
        for u in range(2):
            o = swizzle((start + m) * 2 * CH + 32 * s + 16 * u, 2 * CH) // 2
            out[m, 8 * u:8 * u + 8] = st[o:o + 8]
    return out


@pytest.mark.parametrize("H,W,CH,R", [(4, 128, 16, 4), (3, 256, 32, 1), (2, 128, 32, 2),      # k_conv3x3_rows
                                      (5, 9, 16, 0), (3, 100, 32, 0), (7, 129, 32, 0), (1, 1, 16, 0)])  # its FLAT form
def test_windows_give_the_convolution(plan, H, W, CH, R):
    rng = np.random.default_rng(H * W)
    Cin, BN = 2 * CH, 16
    x = rng.integers(-3, 4, (1, H, W, Cin)).astype(float)
    w = rng.integers(-2, 3, (BN, 9, Cin)).astype(float)
    pad = np.pad(x[0], ((1, 1), (1, 1), (0, 0)))
    want = sum(np.einsum("yxc,oc->yxo", pad[t // 3:t // 3 + H, t % 3:t % 3 + W], w[:, t]) for t in range(9))
    flat = R == 0
    bw, rows = plan("t", [(H, W, 2)])[0] if flat else (BM, R)
    pitch, c = bw + 2, cfg(BN, 1 if flat else R, CH)
    got = np.full((H, W, BN), np.nan)
    for y0 in range(0, H, rows):
        for x0 in range(0, W, bw):
            acc = np.zeros((1 if flat else R, BM, BN))
            for kc in range(Cin // CH):
                st = stage(x, 0, x0 - 1, y0 - 1, pitch, rows + 2, kc * CH, CH, c["A"])
                for s in range(CH // 16):
                    for tap in range(9):
                        ci = kc * CH + 16 * s
                        for r in range(acc.shape[0]):
                            acc[r] += window(st, (r + tap // 3) * pitch + tap % 3, CH, s) @ w[:, tap, ci:ci + 16].T
            for r in range(acc.shape[0]):
                for m in range(BM):
                    my, mx = (m // pitch, m % pitch) if flat else (r, m)
                    if mx < bw and my < rows and y0 + my < H and x0 + mx < W:
                        got[y0 + my, x0 + mx] = acc[r, m]
    assert np.array_equal(got, want)  # integers; a NaN would be a pixel never written or a window outside its box
