"""The bilateral grid method (grid_gpu) against the reference's own GRID method:
JointBilateral::apply / Bilateral::apply / GaussTransform::apply with GaussTransform::GRID
(src/GaussTransform.cpp:227-290, src/DenseGrid.h).  The splat's atomics add in another
order than the reference's serial loop; everything else follows its arithmetic, so the
results agree to FP32 rounding."""
import numpy as np
import pytest

import oracle
from imagestack_b200 import synth

pytestmark = pytest.mark.gpu

RTOL = 1e-5


def rel_err(a, b, floor_frac=1e-6):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    floor = max(np.abs(b).max() * floor_frac, 1e-30)
    return float((np.abs(a - b) / np.maximum(np.abs(b), floor)).max())


def test_grey_joint_bilateral_d3_matches_reference_grid(gpu):
    rgb = synth.image(256, 192, 3, rects=8, seed=31)
    grey = synth.luminance(rgb)
    guide = synth.luminance(synth.image(256, 192, 3, rects=8, seed=32))
    ref, _ = oracle.reference_joint_bilateral(grey, guide, 8.0, 0.1, method="grid")
    out = grey.copy()
    gpu.JointBilateral.apply(out, guide, 8.0, 8.0, 0.0, 0.1, method="grid_gpu")
    assert rel_err(out, ref) <= RTOL


def test_rgb_bilateral_d5_matches_reference_grid(gpu):
    img = synth.image(96, 64, 3, rects=6, seed=33)
    ref, _ = oracle.reference_bilateral(img, 6.0, 0.2, method="grid")
    out = img.copy()
    gpu.Bilateral.apply(out, 6.0, 6.0, 0.0, 0.2, method="grid_gpu")
    assert rel_err(out, ref) <= RTOL


def test_gauss_transform_grid_with_other_slice_positions(gpu):
    rng = np.random.default_rng(34)
    splat = rng.uniform(0, 8, (2, 1, 40, 50)).astype(np.float32)
    slice_ = rng.uniform(-1, 9, (2, 1, 40, 50)).astype(np.float32)   # other positions
    vals = np.concatenate([rng.uniform(-1, 1, (2, 1, 40, 50)),
                           np.ones((1, 1, 40, 50))]).astype(np.float32)
    sig = [1.5, 0.75]
    ref, _ = oracle.reference_gauss_transform(slice_, splat, vals, sig, method="grid")
    out = gpu.GaussTransform.apply(slice_, splat, vals, sig, method="grid_gpu")
    assert out.shape == ref.shape
    # signed values cancel: errors are measured against 1 % of the output's magnitude
    assert rel_err(out, ref, floor_frac=1e-2) <= RTOL


def test_grid_method_limits(gpu):
    img = synth.image(32, 24, 7, rects=2, seed=35)   # d = 9 positions: too many corners
    with pytest.raises(gpu.PgpuError) as e:
        gpu.Bilateral.apply(img, 4.0, 4.0, 0.0, 0.2, method="grid_gpu")
    assert e.value.code == gpu.ERR_UNSUPPORTED


def grid_in_64_bits(pos, val, slice_pos):
    """The bilateral grid (src/DenseGrid.h) over columns of pos (d, n) in FP64: cells by the
    single-precision positions, multilinear splat, two [1 2 1]/4 passes, multilinear slice."""
    d = pos.shape[0]
    sf = np.float32(np.sqrt(np.float32(1.0 / 3 + 1.0)))
    both = np.concatenate([pos, slice_pos], 1) * sf
    low = both.min(1)
    sizes = [int(np.ceil(s)) + 1 for s in both.max(1) - low]

    def corners(p):
        f = p * sf - low[:, None]
        cell = np.floor(f)
        frac = (f - cell).astype(np.float64)
        for corner in range(1 << d):
            w, at = np.ones(p.shape[1]), []
            for j in range(d):
                up = (corner >> j) & 1
                w = w * (frac[j] if up else 1.0 - frac[j])
                at.append(np.minimum(cell[j].astype(int) + up, sizes[j] - 1))   # past the end: weight 0
            yield tuple(at), w

    rows = np.zeros(sizes + [val.shape[0]])
    for at, w in corners(pos):
        np.add.at(rows, at, w[:, None] * val.T)
    for j in range(d):
        for _ in range(2):
            pad = np.pad(rows, [(1, 1) if k == j else (0, 0) for k in range(d + 1)])
            take = lambda o: np.take(pad, np.arange(sizes[j]) + o, axis=j)
            rows = 0.25 * take(0) + 0.5 * take(1) + 0.25 * take(2)
    return sum(rows[at] * w[:, None] for at, w in corners(slice_pos)).T


@pytest.mark.gpu
@pytest.mark.parametrize("d,vd,n,m", [(1, 2, 1, 1), (1, 2, 4097, 3), (2, 2, 255, 1030), (3, 2, 1025, 257),
                                      (2, 4, 514, 77), (3, 3, 300, 301), (4, 2, 999, 64), (5, 1, 130, 1)])
def test_grid_kernels_match_64_bits(gpu, d, vd, n, m):
    """Runs of four points cut by the end of the row, cells in pairs (two values, d <= 3), single
    cells per dimension, and slices elsewhere and at the splat's own points."""
    rng = np.random.default_rng(7 * d + vd)
    pos = rng.uniform(0, 4, (d, n)).astype(np.float32)
    pos[:, n // 2:] = pos[:, :n - n // 2]      # points that share cells
    if d > 1:
        pos[d - 1] = 1.25                      # one cell along this dimension
    val = rng.uniform(0, 1, (vd, n)).astype(np.float32)
    other = rng.uniform(0, 4, (d, m)).astype(np.float32)
    if d > 1:
        other[d - 1] = 1.25
    for q in (None, other):
        out = gpu.GaussTransform.apply(None if q is None else q.reshape(d, 1, -1), pos.reshape(d, 1, n),
                                       val.reshape(vd, 1, n), [1.0] * d, method="grid_gpu").reshape(vd, -1)
        ref = grid_in_64_bits(pos, val, pos if q is None else q)
        assert np.abs(out - ref).max() <= 1e-5 * np.abs(ref).max()
