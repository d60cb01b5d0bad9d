"""Results written into page-locked buffers that start anywhere: every scan's buffers are slices of arrays
that hold the whole batch's, aligned to nothing but their type, and the sizes lie about a label tile's. They equal
the results copied through pageable buffers, and no byte outside a slice changes."""
import numpy as np
import pytest

import lidar_gb300 as lp
import lp_testlib as T

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 1023, 1024, 1025, 2047, 5000, 17, 4099]
GUARD = 0xA5


@pytest.mark.parametrize("noise", [0, 1])
@pytest.mark.parametrize("shift", [0, 1, 2, 3, 5, 31])
def test_slices_at_any_offset(ctx, noise, shift):
    pts, ring, cfg = T.synth_scan(3, 8)[:3]
    pick = [np.sort(np.random.default_rng(n).permutation(len(pts))[:n]) for n in SIZES]
    xs = [np.ascontiguousarray(pts[k]) for k in pick]
    rings = [np.ascontiguousarray(ring[k]) for k in pick]
    pipe = lp.PipelineConfig.default(enable_noise_removal=noise)
    want = lp.process_batch(ctx, xs, pipe, [cfg] * len(xs), rings)

    caps = [n // 3 + 2 for n in SIZES]
    hcap = [n + c for n, c in zip(SIZES, caps)]
    box = np.dtype([("w", np.uint32, 19), ("pad", np.uint32)])

    def guarded(counts, dt):
        """One page-locked array for slices of these lengths, `shift` elements in and apart."""
        a = lp.pinned_empty((sum(counts) + shift * (len(counts) + 1)) * np.dtype(dt).itemsize, np.uint8)
        a[...] = GUARD
        v, at, out = a.view(dt), shift, []
        for n in counts:
            out.append(v[at:at + n])
            at += n + shift
        return a, out

    one = [c + 1 for c in caps]
    arrays = {"noise": guarded(SIZES, np.uint8), "seg": guarded(SIZES, np.uint32), "cl": guarded(SIZES, np.int32),
              "hoff": guarded(one, np.uint32), "hidx": guarded(hcap, np.int32), "zmin": guarded(caps, np.float32),
              "zmax": guarded(caps, np.float32), "c": guarded(caps, box), "p": guarded(caps, box)}
    assert box.itemsize == lp.ctypes.sizeof(lp.BoundingBox)

    class Buf:
        pass

    bufs = []
    for j in range(len(SIZES)):
        b = Buf()
        b.v = {k: a[1][j] for k, a in arrays.items()}
        b.seg = b.v["seg"]
        g = lambda k: lp.ptr(b.v[k])
        b.out = lp.ScanOutput(g("noise"), g("seg"), g("cl"), caps[j], hcap[j], g("hoff"), g("hidx"), g("zmin"),
                              g("zmax"), g("c"), g("p"), 0, 0, 0, 0)
        bufs.append(b)
    px = [lp.pinned_copy(x) for x in xs]
    pr = [lp.pinned_copy(r) for r in rings]
    lp.process_batch(ctx, px, pipe, [cfg] * len(xs), pr, outputs=bufs, raw=True)

    used = {k: [] for k in arrays}
    for j, (b, w) in enumerate(zip(bufs, want)):
        k, h = b.out.n_clusters, b.out.n_hull_indices
        assert (k, b.out.n_obstacles, h) == (w.n_clusters, w.n_obstacles, len(w.hull_indices)), f"scan {j}"
        boxes = lambda a: np.array([np.frombuffer(bytes(x), np.uint32)[:19] for x in a], np.uint32).reshape(-1, 19)
        for name, n, ref in [("noise", SIZES[j], w.noise_labels), ("seg", SIZES[j], w.seg_labels),
                             ("cl", SIZES[j], w.cluster_labels), ("hoff", k + 1, w.hull_offsets),
                             ("hidx", h, w.hull_indices), ("zmin", k, w.z_min), ("zmax", k, w.z_max)]:
            assert np.array_equal(b.v[name][:n], ref), f"scan {j} {name}"
        assert np.array_equal(b.v["c"]["w"][:k], boxes(w.obb_calipers)), f"scan {j} calipers"
        assert np.array_equal(b.v["p"]["w"][:k], boxes(w.obb_pca)), f"scan {j} pca"
        for name, n in [("noise", SIZES[j]), ("seg", SIZES[j]), ("cl", SIZES[j]), ("hoff", k + 1), ("hidx", h),
                        ("zmin", k), ("zmax", k), ("c", k), ("p", k)]:
            used[name].append(b.v[name][:n])
    for name, (a, _) in arrays.items():  # nothing outside the results was written
        for v in used[name]:
            v.view(np.uint8)[...] = GUARD
        assert (a == GUARD).all(), name
