"""Queries of one handle from two host threads at once, which the contract
forbids: their own answers may be wrong, the ones of later queries may not."""
import threading

import numpy as np
import pytest
import torch

from bulbit_b200 import abi, lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [abi.BBG_TRAVERSAL_WIDE, abi.BBG_TRAVERSAL_ORDERED])
def test_queries_after_overlapping_ones(mode):
    acc = lib.GpuAccel(scenes.triangle_soup(50_000, seed=6, sigma=0.03))
    closest, short = scenes.soup_rays(150_001, seed=9)
    acc.set_traversal(abi.BBG_TRAVERSAL_REFERENCE)
    ref, occ = acc.intersect(closest), acc.intersect_any(short)
    acc.set_traversal(mode)

    def queries(rays, n):
        stream = torch.cuda.Stream()
        out = torch.empty((n, 4), device="cuda")
        for _ in range(60):
            acc.intersect_device(rays[:n], out, stream.cuda_stream)

    rays = torch.from_numpy(closest).cuda()
    torch.cuda.synchronize()
    # Different sizes, so the two launches differ in their number of blocks.
    threads = [threading.Thread(target=queries, args=(rays, n)) for n in (150_001, 20_000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for _ in range(2):
        got = acc.intersect(closest)
        assert np.array_equal(got[1].view(np.uint32), ref[1].view(np.uint32))
        assert np.array_equal(got[0] >= 0, ref[0] >= 0)
        assert np.array_equal(acc.intersect_any(short), occ)
    acc.close()
