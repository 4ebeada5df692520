"""Renders of different sizes from two host threads at the same time, both through the
depth-ordered tile lists: every one succeeds with the lists that it gives alone (a
launch limit set for one size must not reach the other's launch)."""
import threading

import pytest
import torch

import gsplatcu as gsc
from test_gpu_tile_lists import _inputs

pytestmark = pytest.mark.gpu

RENDERS = 60


def _render(s, W, H):
    out = gsc.splat_weight(H, W, 1, s["us"], s["cinv"], s["alphas"], s["depths"].clone(), s["feats"],
                           s["areas"].clone())
    return out[3], out[4]


def test_two_sizes_from_two_threads(cuda_ok):
    sizes = [(1920, 1080), (3840, 2160)]
    scenes = [_inputs(20000, W, H, seed=W, keys=9000, patches=4_000_000) for W, H in sizes]
    want = [_render(s, W, H) for s, (W, H) in zip(scenes, sizes)]
    torch.cuda.synchronize()
    wrong, together = [], threading.Barrier(2)

    def work(s, W, H, ref):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                together.wait()
                for _ in range(RENDERS):
                    got = _render(s, W, H)
                    if not all(torch.equal(a, b) for a, b in zip(got, ref)):
                        wrong.append((W, H))
        except Exception as e:  # reported by the assertion below
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(s, W, H, r))
               for s, (W, H), r in zip(scenes, sizes, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
