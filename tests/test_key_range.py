"""Lattices whose keys lie at the ends of what a compact key's fields hold, and beyond: the
results have to be those of the reference's int16 keys wherever the positions lie."""
import ctypes as C

import numpy as np
import pytest

import oracle
from imagestack_b200 import synth
from test_gpu_parity import RTOL_FP32, rel_err

pytestmark = pytest.mark.gpu

# bits of a quotient's field by d (64-bit keys to d = 7, 128 above), and the quotients where
# compact keys end
FIELD_BITS = {5: 12, 6: 10, 7: 8, 9: 9, 12: 9, 13: 7, 15: 7, 16: 7}


def elevation(d):
    """The linear map of positions to the lattice's d+1 coordinates (src/Permutohedral.h:293-299)."""
    sf = np.empty(64, np.float32)
    oracle._load_oracle().lo_scale_factors(d, sf)
    e = np.zeros((d + 1, d))
    e[d, d - 1] = -d * sf[d - 1]
    for i in range(d - 1, 0, -1):
        e[i] = e[i + 1]
        e[i, i - 1] -= i * sf[i - 1]
        e[i, i] += (i + 2) * sf[i]
    e[0] = e[1]
    e[0, 0] += 2 * sf[0]
    return e


def positions(coords):
    """Positions whose lattice coordinates are `coords` (rows of d+1 numbers of sum zero)."""
    d = coords.shape[1] - 1
    return np.ascontiguousarray((coords @ np.linalg.pinv(elevation(d)).T).astype(np.float32))


def check(gpu, pos, val):
    ref = oracle.oracle_lattice(pos, val)
    got = gpu.lattice_dump(pos, val)
    for k in ("keys", "replay_vtx", "replay_w"):
        np.testing.assert_array_equal(got[k], getattr(ref, k))
    for k in ("splat", "blur", "out"):
        assert rel_err(got[k], getattr(ref, k)) <= RTOL_FP32


@pytest.mark.parametrize("step", [-1, 0, 1, 2])
@pytest.mark.parametrize("d", sorted(FIELD_BITS))
def test_quotients_at_the_ends_of_the_fields(gpu, d, step):
    """Points whose greedy quotients are the largest a compact key takes, and one or two
    more, along every coordinate and at both ends."""
    rng = np.random.default_rng(10 * d + step)
    top = (1 << (FIELD_BITS[d] - 1)) - 3 + step
    q = np.zeros((2 * (d + 1), d + 1))
    for i in range(d + 1):
        q[2 * i, i], q[2 * i, (i + 1) % (d + 1)] = top, -top
        q[2 * i + 1, i], q[2 * i + 1, (i + 2) % (d + 1)] = -top, top
    off = rng.uniform(-0.9, 0.9, (20, 2 * (d + 1), d + 1)) * (d + 1)
    coords = (q * (d + 1) + off - off.mean(2, keepdims=True)).reshape(-1, d + 1)
    val = rng.uniform(0, 1, (len(coords), 4)).astype(np.float32)
    check(gpu, positions(coords), val)


def points_around(c, r, i, rank_i, rng, n):
    """n points of simplices that have vertex c (d+1 coordinates, remainder r), coordinate i
    of rank rank_i in them (src/Permutohedral.h:367-369)."""
    d = len(c) - 1
    coords = np.empty((n, d + 1))
    for k in range(n):
        rank = rng.permutation(d + 1)
        j = int(np.flatnonzero(rank == rank_i)[0])
        rank[j], rank[i] = rank[i], rank_i
        step = np.array([np.where(rank <= d - s, s, s - (d + 1)) for s in range(d + 1)])
        coords[k] = c - step[r] + rng.dirichlet(np.ones(d + 1)) @ step
    return positions(coords)


@pytest.mark.parametrize("mode,ends", [
    # neighbour down of remainder 1, quotient 63: quotient 64 would carry into remainder 16
    ("both", ((1, 63, -56, 15), (16, -64, 56, 1))),
    # neighbour up of remainder 15, quotient -64: quotient -65 would borrow from remainder 16
    ("half", ((15, -64, 56, 2), (0, 63, -56, 16))),
])
def test_no_neighbour_across_a_field_of_sixteen_dimensions(gpu, monkeypatch, mode, ends):
    """Two far points with a vertex each whose keys differ by what a carry out of coordinate
    11's 7-bit field would make of the first one's neighbour along that axis."""
    monkeypatch.setenv("PGPU_NBR", mode)
    d, i = 16, 11
    rng = np.random.default_rng(1)
    e = elevation(d)
    pos = []
    for r, q_i, q_d, rank_i in ends:
        q = np.zeros(d + 1)
        q[i], q[d] = q_i, q_d
        q[:int(q.sum() + r)] = -1   # the coordinates' sum is zero
        c = q * (d + 1) + r
        assert c.sum() == 0
        p = points_around(c, r, i, rank_i, rng, 4000)
        keys, _ = oracle.oracle_simplex(p)
        has = (keys[:, r] == c[:d]).all(1)
        # the greedy point's quotients are 62 at most
        has &= np.abs(np.rint(p.astype(np.float64) @ e.T / (d + 1))).max(1) <= 62
        assert has.sum() >= 3
        pos.append(p[has][:3])
    pos = np.concatenate(pos)
    check(gpu, pos, rng.uniform(0.5, 1, (len(pos), 4)).astype(np.float32))


def transform_into(gpu, slice_pos, splat_pos, values, out):
    """pgpu_gauss_transform of device memory with an output of the caller's choice, which may
    be one of the inputs."""
    d = splat_pos.shape[0]
    views = [gpu._view(t, "view")[0] for t in (slice_pos, splat_pos, values, out)]
    opt = gpu._options(gpu.MEM_DEVICE, "fp32", stream=gpu._torch_stream(values))
    gpu._check(gpu.lib().pgpu_gauss_transform(C.byref(views[0]), C.byref(views[1]), C.byref(views[2]),
                                              (C.c_float * d)(*[1.0] * d), d, C.byref(views[3]), C.byref(opt)))


@pytest.mark.parametrize("into", ["new", "values", "slice"])
@pytest.mark.parametrize("d,reach", [(1, 18000.0), (3, 9000.0), (5, 4500.0), (7, 600.0), (9, 2000.0), (16, 400.0)])
def test_slice_positions_out_of_the_compact_range(gpu, d, reach, into):
    """The splat's positions fit compact keys, a few of the slice's do not (they stay within the
    reference's int16 keys) and have no vertices; the output may be one of the inputs."""
    import torch
    rng = np.random.default_rng(7 * d)
    n = 40000 + len(into)   # images of their own shape: nothing is known of them
    pos = (rng.integers(0, 4, (n, 1)) * 3.0 + rng.normal(0, 0.4, (n, d))).astype(np.float32)
    other = (pos[::-1] + rng.normal(0, 0.3, (n, d))).astype(np.float32)
    other[n - 700::7, d - 1] += np.linspace(-reach, reach, 100).astype(np.float32)
    val = rng.uniform(0, 1, (n, d)).astype(np.float32)[:, :min(d, 8)]
    if into == "slice" and val.shape[1] < d:
        pytest.skip("as many values as positions, to write over them")
    ref = oracle.oracle_lattice(pos, val, slice_pos=other).out
    planar = lambda a: torch.from_numpy(np.ascontiguousarray(a.T).reshape(a.shape[1], 1, n)).cuda()
    ts, tp, tv = planar(other), planar(pos), planar(val)
    transform_into(gpu, tp, tp, tv, torch.empty_like(tv))   # the table's size is learned
    out = {"new": torch.empty_like(tv), "values": tv, "slice": ts}[into]
    transform_into(gpu, ts, tp, tv, out)
    torch.cuda.synchronize()
    assert rel_err(out.cpu().numpy().reshape(-1, n).T, ref) <= RTOL_FP32
    assert gpu.last_stats()["retries"] == 0


@pytest.mark.parametrize("d,sign", [(1, 1), (1, -1), (3, 1), (3, -1), (4, 1)])
def test_slice_positions_at_the_ends_of_int16(gpu, d, sign):
    """Vertices near one end of int16 and slice positions near both: keys that wrap around in
    the reference's shorts wrap here too, and positions beyond int16 fail the call."""
    rng = np.random.default_rng(3 * d + sign)
    top = 32767 // (d + 1)
    def at(q0, n):
        q = np.zeros((n, d + 1))
        q[:, 0], q[:, d] = q0, -q0
        off = rng.uniform(-0.45, 0.45, (n, d + 1)) * (d + 1)
        return positions(q * (d + 1) + off - off.mean(1, keepdims=True))
    pos = at(sign * (top - 3), 500)
    val = rng.uniform(0, 1, (500, 2)).astype(np.float32)
    other = np.concatenate([at(sign * (top - 3), 300), at(sign * (top - 1), 300), at(-sign * (top - 1), 300)])
    ref = oracle.oracle_lattice(pos, val, slice_pos=other).out
    planar = lambda a: np.ascontiguousarray(a.T).reshape(a.shape[1], 1, len(a))
    out = gpu.GaussTransform.apply(planar(other), planar(pos), planar(val), [1.0] * d)
    assert rel_err(out.reshape(2, -1).T, ref) <= RTOL_FP32
    with pytest.raises(gpu.PgpuError):
        far = at(sign * (top + 3), 10)
        gpu.GaussTransform.apply(planar(far), planar(pos), planar(val), [1.0] * d)


def test_images_too_large_for_compact_keys_start_on_wide_keys(gpu):
    """Images whose pixel coordinates alone leave the fields' range: no rerun, at the first call
    of a shape, for any place of the large coordinate."""
    rng = np.random.default_rng(4)
    for k, (w, h, sx, sy) in enumerate([(402, 90, 1.0, 9.0), (403, 91, 1.0, 9.0), (90, 410, 9.0, 1.0), (300, 50, 1.0, 8.0)]):
        guide = rng.uniform(0, 1, (5, h, w)).astype(np.float32)   # nearly no vertex is shared
        im = rng.uniform(0, 1, (2, h, w)).astype(np.float32)
        out = im.copy()
        gpu.JointBilateral.apply(out, guide, sx, sy, 0.0, 0.05)
        assert k == 0 or gpu.last_stats()["retries"] == 0
        pos, val = oracle.bilateral_points(im, guide, sx, 0.05, sigma_s_y=sy)
        ref = oracle.oracle_lattice(pos, val).out
        norm = (ref[:, :2] / ref[:, 2:]).reshape(h, w, 2).transpose(2, 0, 1)
        assert rel_err(out, norm) <= RTOL_FP32


def test_an_image_that_needs_wide_keys_does_not_mark_its_shape(gpu):
    """Images of one shape: after one that needs int16 lanes the next starts on them; after one
    that does not, or one that fails the call, compact keys are tried first (a rerun where
    they do not fit)."""
    rng = np.random.default_rng(3)
    noise = rng.uniform(0, 1, (3, 61, 83)).astype(np.float32)   # nearly no vertex is shared, so
    near, far = noise * np.float32(16.0), noise * np.float32(3000.0)   # both need the same table
    bad = near.copy()
    bad[1, 30, 40] = np.nan

    def reruns(img):
        out = img.copy()
        gpu.Bilateral.apply(out, 6.0, 6.0, 0.0, 0.8)
        pos, val = oracle.bilateral_points(img, img, 6.0, 0.8)
        ref = oracle.oracle_lattice(pos, val).out
        norm = (ref[:, :3] / ref[:, 3:4]).reshape(61, 83, 3).transpose(2, 0, 1)
        assert rel_err(out, norm) <= RTOL_FP32
        return gpu.last_stats()["retries"]

    reruns(near)   # the table's size is learned
    for _ in range(2):
        assert reruns(near) == 0   # (on int16 lanes the second time round)
        assert reruns(near) == 0
        with pytest.raises(gpu.PgpuError):
            gpu.Bilateral.apply(bad, 6.0, 6.0, 0.0, 0.8)
        assert reruns(near) == 0
        assert reruns(far) >= 1
        assert reruns(far) == 0


@pytest.mark.parametrize("graph", [False, True])
def test_queued_batch_with_an_image_known_to_need_wide_keys(gpu, graph):
    """Queued batches in which one image needs int16 lanes, unknown and known: the others stay
    on the tile splat of compact keys, and every result lands in its own output."""
    imgs = [synth.image(w, h, 3, rects=6, seed=w) for w, h in ((150, 91), (98, 133), (64, 65), (77, 60))]
    imgs[1] = (imgs[1] * 3000).astype(np.float32)   # colours thousands of sigmas apart
    fw, cs = [6.0, 5.0, 8.0, 7.0], [0.1, 0.8, 0.2, 0.3]
    expect = [im.copy() for im in imgs]
    for im, f, c in zip(expect, fw, cs):
        gpu.Bilateral.apply(im, f, f, 0.0, c, payload="fp64")
    gpu.Bilateral.apply(imgs[1].copy(), fw[1], fw[1], 0.0, cs[1])   # known from here on
    for _ in range(3):
        out = [np.empty_like(im) for im in imgs]
        gpu.bilateral_batch_submit(imgs, fw, cs, outputs=out, graph=graph).wait()
        assert gpu.last_stats()["tiled"] >= 3 and gpu.last_stats()["retries"] == 0
        for a, b in zip(out, expect):
            assert rel_err(a, b, floor_frac=1e-2) <= RTOL_FP32
    # nothing known of these shapes: the first batch finds out as it completes
    imgs = [np.ascontiguousarray(im[:, 1 + int(graph):]) for im in imgs]
    outs = [[np.empty_like(im) for im in imgs] for _ in range(3)]
    tickets = [gpu.bilateral_batch_submit(imgs, fw, cs, outputs=out, graph=graph) for out in outs]
    for t in tickets:
        t.wait()
    expect = [im.copy() for im in imgs]
    for im, f, c in zip(expect, fw, cs):
        gpu.Bilateral.apply(im, f, f, 0.0, c, payload="fp64")
    for out in outs:
        for a, b in zip(out, expect):
            assert rel_err(a, b, floor_frac=1e-2) <= RTOL_FP32


@pytest.mark.parametrize("rows", ["slot", "vertex"])
@pytest.mark.parametrize("mode", ["direct", "tile"])
@pytest.mark.parametrize("c,w,h", [(1, 257, 33), (2, 16, 16), (3, 129, 66), (4, 33, 255), (5, 40, 47), (5, 300, 1)])
def test_int16_lane_splats_of_images(gpu, monkeypatch, c, w, h, mode, rows):
    """Both splats on int16 lanes over whole and ragged tiles, and their dumps."""
    monkeypatch.setenv("PGPU_KEYS", "wide")
    monkeypatch.setenv("PGPU_SPLAT", mode)
    monkeypatch.setenv("PGPU_ROWS", rows)
    img = synth.image(w, max(h, 2), c, rects=5, seed=w + h)[:, :h]
    pos, val = oracle.bilateral_points(img, img, 3.0, 0.15)
    if h > 1:
        out = img.copy()
        gpu.Bilateral.apply(out, 3.0, 3.0, 0.0, 0.15)
        ref = oracle.oracle_lattice(pos, val).out
        norm = (ref[:, :c] / ref[:, c:]).reshape(h, w, c).transpose(2, 0, 1)
        assert rel_err(out, norm) <= RTOL_FP32
        assert gpu.last_stats()["tiled"] == (1 if mode == "tile" else 0)
    check(gpu, pos, val)


def test_messages_name_the_image_of_the_batch(gpu):
    """The image that fails a batch is named by its place in the caller's list, also where the
    passes took the images in another order."""
    imgs = [synth.image(90, 70, 3, rects=4, seed=s) for s in range(4)]
    imgs[0] = (imgs[0] * 3000).astype(np.float32)   # int16 lanes
    imgs[2][1, 5, 6] = np.nan
    fw, cs = [5.0, 5.5, 6.0, 6.5], [0.8, 0.2, 0.3, 0.4]
    for _ in range(2):
        with pytest.raises(gpu.PgpuError, match="image 2:"):
            gpu.bilateral_batch([im.copy() for im in imgs], fw, cs)
        with pytest.raises(gpu.PgpuError, match="image 2:"):
            gpu.bilateral_batch_submit([im.copy() for im in imgs], fw, cs).wait()
