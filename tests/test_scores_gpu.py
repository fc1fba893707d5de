"""Edges of the post-processing kernels: cluster sizes around the blocks of the centroid sums, absent
labels, the silhouette's runs of clusters."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _labels(sizes, rng):
    """Labels c repeated sizes[c] times, shuffled, with some -1 among them."""
    lab = np.concatenate([np.full(s, c, np.int32) for c, s in enumerate(sizes)] + [np.full(57, -1, np.int32)])
    return rng.permutation(lab)


@pytest.mark.parametrize("ndim", [1, 2, 5, 10])
@pytest.mark.parametrize("sizes", [[1], [3, 0, 0, 1, 4], [127, 128, 129, 256, 257, 1, 1000], [5000, 2], [40] * 300])
def test_centroids_by_cluster_size(gpu_context, sizes, ndim):
    rng = np.random.default_rng(len(sizes) + ndim)
    lab = _labels(sizes, rng)
    c = rng.normal(0, 10, size=(ndim, lab.size)).astype(np.float32)
    cen, got = gpu_context.cluster_centroids(c, lab)
    np.testing.assert_array_equal(got, sizes)
    for k, s in enumerate(sizes):
        for d in range(ndim):
            acc = np.float32(0)
            for v in c[d, lab == k]:
                acc = np.float32(acc + v)
            if s:
                assert np.float32(acc / np.float32(s)).view(np.uint32) == cen[k, d].view(np.uint32)


@pytest.mark.parametrize("labels", [np.array([-1], np.int32), np.array([0], np.int32), np.full(3000, -1, np.int32),
                                    np.array([4999] + [-1] * 4999, np.int32),
                                    np.array([0, 4999] * 2500, np.int32),
                                    np.arange(70000, dtype=np.int32)[::-1].copy()], ids=range(6))
def test_association_map_of_absent_labels(gpu_context, labels):
    import torch
    n = labels.size
    d = torch.from_numpy(labels).cuda()
    off = torch.full((n + 1,), -7, dtype=torch.int32, device="cuda")
    pts = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    nc, nin = gpu_context.get_clusters(d.data_ptr(), n, off.data_ptr(), pts.data_ptr())
    keep = np.nonzero(labels >= 0)[0]
    assert (nc, nin) == (labels.max() + 1, keep.size)
    want = np.concatenate([[0], np.cumsum(np.bincount(labels[keep], minlength=n))]).astype(np.int32)
    np.testing.assert_array_equal(off.cpu().numpy(), want)
    np.testing.assert_array_equal(pts.cpu().numpy()[:nin], keep[np.argsort(labels[keep], kind="stable")])


@pytest.mark.parametrize("ndim", [1, 2, 3, 6, 9])
@pytest.mark.parametrize("sizes", [[2], [1, 1, 2], [255, 1, 256, 0, 257, 3], [5] * 200, [3000, 1, 700]])
def test_silhouette_runs_of_clusters(gpu_context, sizes, ndim):
    import torch
    rng = np.random.default_rng(len(sizes) * 7 + ndim)
    lab = _labels(sizes, rng)
    c = rng.normal(0, 3, size=(ndim, lab.size)).astype(np.float32)
    ref, ref_mean = O.silhouette(c, lab)
    dc, dl = torch.from_numpy(c).cuda(), torch.from_numpy(lab).cuda()
    per = torch.empty(lab.size, device="cuda")
    torch.cuda.synchronize()
    mean = gpu_context.silhouette_device(dc.data_ptr(), dl.data_ptr(), ndim, lab.size, per.data_ptr())
    got = per.cpu().numpy()
    nan = np.isnan(ref)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.uint32), ref[~nan].view(np.uint32))
    assert np.float32(mean).view(np.uint32) == np.float32(ref_mean).view(np.uint32) or nan.all()
