"""Host threads that run the iterative solvers at the same time, each with its own frame size,
workspace and stream: every call succeeds and gives the result that it gives alone."""
import threading

import numpy as np
import pytest

import mvs_b200 as M
from test_tgv2_persistent_gpu import _setup
from test_tgv2_sparse_gpu import sparse_case

pytestmark = pytest.mark.gpu

SIZES = [(640, 480), (97, 73), (320, 240)]


def _denoise(cuda, w, h):
    import torch
    ref, depth, _ = sparse_case(w, w, h)
    ref, depth = torch.from_numpy(ref).to(cuda), torch.from_numpy(depth).to(cuda)
    ws = torch.empty(M.tvl1_workspace_bytes(w, h) // 8 + 1, dtype=torch.int64, device=cuda)
    out = torch.empty_like(depth)

    def call(stream):
        out.copy_(depth)
        M.tvl1_denoise(ref, out, 0.4, 8.0, M.tvl1_params(niters=60), ws, stream=stream)
        return out
    return call


def _sparse(cuda, w, h):
    import torch
    ref, depth, sp = (torch.from_numpy(a).to(cuda) for a in sparse_case(w, w, h))
    ws = torch.empty(M.tgv2_sparse_workspace_bytes(w, h) // 8 + 1, dtype=torch.int64, device=cuda)
    out = torch.empty_like(depth)

    def call(stream):
        M.tgv2_sparse(ref, depth, sp, 6.0, out, ws, 60, stream=stream)
        return out
    return call


def _tgv2(cuda, w, h):
    s = _setup(cuda, w, h, 4, seed=w)
    u = s["start"].clone()

    def call(stream):
        u.copy_(s["start"])
        M.tgv2_run(s["ref"], s["srcs"], s["K"], s["iK"], s["Rs"], s["ts"], M.tgv2_params(niters=60, warps=1), u,
                   u_from_input=True, workspace=s["ws"], stream=stream)
        return u
    return call


@pytest.mark.parametrize("make", [_denoise, _sparse, _tgv2])
def test_threads_with_different_frame_sizes(cuda, make):
    import torch
    sizes = [(320, 240), (97, 73), (160, 120)] if make is _tgv2 else SIZES
    calls = [make(cuda, w, h) for w, h in sizes]
    alone = []
    for c in calls:
        r = c(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        alone.append(r.cpu().numpy())
    together, errors = [None] * len(calls), []
    start = threading.Barrier(len(calls))

    def work(k):
        try:
            st = torch.cuda.Stream()
            start.wait()
            with torch.cuda.stream(st):
                for _ in range(60):
                    r = calls[k](st.cuda_stream)
                st.synchronize()
                together[k] = r.cpu().numpy()
        except Exception as e:   # reported by the test's thread
            errors.append((sizes[k], e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(alone, together):
        np.testing.assert_array_equal(a, b)
