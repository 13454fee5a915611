"""Region growing on the GPU (reference: torch_points_kernels/cluster.py, a numba traversal on
the CPU there).  The neighbour search is the packed ball query; the clusters come from label
propagation on the device (tpk_grow_labels_begin, _push) instead of a sequential traversal."""
import ctypes
from typing import List

import torch

from . import _lib
from .torchpoints import ball_query_partial_dense

# Scratch of the labels by trees is as large as the lists: beyond this the lists are walked in every round instead, so
# that lists which fill half of the memory still get labels (160000 points, 16 slots: 38 rounds of 15 us for 130 us).
_MOST_SCRATCH = 8 << 30


def cluster_labels(neighbours):
    """neighbours: (N, nsample) int64 CUDA tensor of neighbour lists (-1 ends a list).  Returns
    (N,) int32 labels: labels[v] = smallest index that reaches v along the lists = seed of the
    cluster the reference's traversal (cluster.py:8-37) assigns v to."""
    _lib.check_cuda(neighbours, "neighbours")
    if neighbours.dtype != torch.int64:
        raise RuntimeError("neighbours must be an int64 tensor")
    neighbours = neighbours.contiguous()
    n, nsample = neighbours.shape
    if n == 0:
        return torch.empty(0, dtype=torch.int32, device=neighbours.device)
    with _lib.on_device(neighbours):
        stream = _lib.stream_of(neighbours)
        need = _lib.lib().tpk_grow_labels_scratch_bytes(n, nsample)
        if need <= _MOST_SCRATCH:
            # labels go along the lists between trees of points that list each other: a few rounds as a rule
            labels = torch.empty(n, dtype=torch.int32, device=neighbours.device)
            changed = torch.empty(1, dtype=torch.int32, device=neighbours.device)
            scratch = torch.empty((need,), dtype=torch.uint8, device=neighbours.device)
            _lib.call("tpk_grow_labels_begin", n, nsample, _lib.ptr(neighbours), _lib.ptr(scratch), need, stream)
        else:
            labels = torch.arange(n, dtype=torch.int32, device=neighbours.device)
            changed = torch.zeros(1, dtype=torch.int32, device=neighbours.device)
            scratch = None
        # a handful of launches per host check keeps the number of device-to-host reads small
        for _ in range(n):
            if scratch is not None:
                _lib.call("tpk_grow_labels_push", n, 8, _lib.ptr(labels), _lib.ptr(changed), _lib.ptr(scratch), stream)
            else:
                changed.zero_()
                _lib.call("tpk_grow_labels_step", n, nsample, _lib.ptr(neighbours), _lib.ptr(labels),
                          _lib.ptr(changed), 8, stream)
            if int(changed.item()) == 0:
                break
    return labels


def grow_proximity(pos, batch, nsample=16, radius=0.02, min_cluster_size=32):
    """Grow based on proximity only.  Returns the clusters as lists of point indices, ordered by
    their smallest member; the members of a cluster are listed in ascending order (the reference
    lists them in the order its traversal met them: the sets are the same)."""
    assert pos.shape[0] == batch.shape[0]
    pos = pos.float().contiguous()
    neighbours = ball_query_partial_dense(radius, nsample, pos, pos, batch, batch)[0]
    labels = cluster_labels(neighbours)
    order = torch.sort(labels.long(), stable=True).indices  # members ascending inside a label
    seeds, counts = torch.unique_consecutive(labels[order], return_counts=True)
    clusters = []
    start = 0
    order_h, counts_h = order.cpu(), counts.cpu().tolist()
    for c in counts_h:
        if c >= min_cluster_size:
            clusters.append(order_h[start:start + c].tolist())
        start += c
    return clusters


def _segments(rank, sample):
    """Numbers of the runs of equal (rank, sample), ascending.  The ids are compared, not computed with:
    any sorted ids of a sample will do, negative and huge ones too."""
    segment = torch.zeros(rank.shape, dtype=torch.int64, device=rank.device)
    begins = (rank[1:] != rank[:-1]) | (sample[1:] != sample[:-1])
    torch.cumsum(begins, 0, out=segment[1:])
    return segment


def region_grow(
    pos, labels, batch, ignore_labels=[], nsample=16, radius=0.02, min_cluster_size=32
) -> List[torch.Tensor]:
    """Region growing clustering algorithm proposed in
    PointGroup: Dual-Set Point Grouping for 3D Instance Segmentation
    https://arxiv.org/pdf/2004.01658.pdf
    for instance segmentation

    Parameters
    ----------
    pos: torch.Tensor [N, 3]
        Location of the points
    labels: torch.Tensor [N,]
        labels of each point
    ignore_labels:
        Labels that should be ignored, no region growing will be performed on those
    nsample:
        maximum number of neighbours to consider
    radius:
        radius for the neighbour search
    min_cluster_size:
        Number of points above which a cluster is considered valid
    """
    assert labels.dim() == 1
    assert pos.dim() == 2
    assert pos.shape[0] == labels.shape[0]

    unique_labels, label_rank, label_counts = torch.unique(labels, return_inverse=True, return_counts=True)
    unique_labels = unique_labels.cpu()
    kept = [not (l in ignore_labels) for l in unique_labels]
    if unique_labels.is_floating_point():
        kept = [k and l == l for k, l in zip(kept, unique_labels.tolist())]  # (NaN is no label)
    if not any(kept):
        return []
    if batch.shape[0] != pos.shape[0] or batch.numel() != pos.shape[0]:
        raise IndexError("batch of shape %s does not match %d points" % (tuple(batch.shape), pos.shape[0]))
    # One search and one labelling for all labels: the points ordered by label (original order inside a
    # label), every (label, sample) pair a segment of its own.  Lists, seeds and the order of the clusters
    # are those of a search per label, because the order inside a segment is the same.
    rank_h = torch.tensor([sum(kept[:i]) if k else -1 for i, k in enumerate(kept)], dtype=torch.int32)
    left_out = sum(c for c, k in zip(label_counts.tolist(), kept) if not k)
    rank, ind = (t[left_out:] for t in torch.sort(rank_h.to(pos.device)[label_rank], stable=True))
    segment = _segments(rank, batch.reshape(-1)[ind])
    local_pos = pos[ind].float().contiguous()
    neighbours = ball_query_partial_dense(radius, nsample, local_pos, local_pos, segment, segment)[0]
    seeds = cluster_labels(neighbours)
    seeds, order = torch.sort(seeds, stable=True)  # members ascending inside a cluster
    counts = torch.unique_consecutive(seeds, return_counts=True)[1]
    members = ind[order[torch.repeat_interleave(counts >= min_cluster_size, counts, output_size=order.shape[0])]]
    sizes = [c for c in counts.tolist() if c >= min_cluster_size]
    clusters = [members.new_empty(c) for c in sizes]
    if clusters:
        torch.split_with_sizes_copy(members, sizes, 0, out=clusters)  # one launch for all
    return clusters
