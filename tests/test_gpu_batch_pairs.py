"""Batches whose long problems take clusters of two CTAs, in the small form (N <= 1024, two
candidates per thread) and in the large one, alone and beside short problems and wider
clusters; against the single-problem per-iteration form."""
import numpy as np
import pytest

from test_gpu_batch_clusters import check, lists

pytestmark = pytest.mark.gpu


def cluster_sizes(items, sms):
    """CTAs per problem as the batch chooses them: the least makespan m for which every
    problem's smallest sufficient cluster takes at most m and all of them fill at most the
    GPU for m, with a scan slice (2,048 candidates) and 512 rows per CTA and doubling."""
    time_of = [1.0, 0.62, 0.365, 0.23]
    w = [it[0] * max(len(it[1]), 2048) for it in items]
    m = sum(w) / sms
    while True:
        lg = []
        for it, x in zip(items, w):
            k = 0
            while k < 3 and x * time_of[k] > m and len(it[1]) > 2048 << (k + 1) and it[0] > 512 << k:
                k += 1
            lg.append(k)
        load = sum(x * time_of[k] * (1 << k) for x, k in zip(w, lg))
        if load / sms <= m or max(x * time_of[k] for x, k in zip(w, lg)) >= sum(w):
            return [1 << k for k in lg]
        m *= 1.1


@pytest.mark.parametrize("long,others", [((513, 4000, 3), []), ((800, 6000, 3), []), ((1024, 12000, 40), [(300, 900, 3)] * 4),
                                         ((1025, 7100, 3), []), ((1030, 5000, 60), [(200, 900, 2)] * 4),
                                         ((900, 6000, 3), [(2500, 40000, 3)])])
def test_clusters_of_two(long, others):
    import torch
    items = [lists(*long, 1)] + [lists(*o, 2 + i) for i, o in enumerate(others)]
    sizes = cluster_sizes(items, torch.cuda.get_device_properties(0).multi_processor_count)
    assert sizes[0] == 2 and max(sizes) == (8 if others and others[0][0] > 2048 else 2)
    check(items)
