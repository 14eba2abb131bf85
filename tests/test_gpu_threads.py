"""Entry points whose shared memory follows the call's sizes, called at two sizes from two host threads at once: the kernel's
limit is one setting for both."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _pair(calls, n):
    import torch
    err, gate = [], threading.Barrier(2)

    def work(call):
        with torch.cuda.stream(torch.cuda.Stream()):
            gate.wait()
            rc = [call() for _ in range(n)]
            torch.cuda.synchronize()
        err.extend(r for r in rc if r)
    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return err


def test_tc_gemm_at_one_and_two_buffers():
    import torch
    from vulcan.gpu import _lib as K
    L = K.lib()

    def call(Kd):
        A, B, C = torch.ones(128, Kd).cuda(), torch.ones(16, Kd).cuda(), torch.zeros(128, 16).cuda()
        ws = torch.empty(max(L.vk_tc_gemm_ws_floats(128, 16, Kd), 1)).cuda()
        st = torch.zeros(1, dtype=torch.int32).cuda()
        return lambda: L.vk_tc_gemm(128, 16, Kd, K.ptr(A), Kd, 1, K.ptr(B), 0, 1, Kd, None, 0, 0, K.ptr(C), 16, 1,
                                    K.ptr(ws), ws.numel(), K.ptr(st), K.stream())
    assert not _pair([call(16), call(256)], 3000)


@pytest.mark.parametrize("entry", ["counts", "hits"])
def test_selection_of_short_and_long_lists(entry):
    import torch
    from vulcan.gpu import _lib as K
    L = K.lib()
    i64 = lambda *v: torch.tensor(v, dtype=torch.int64).cuda()  # noqa: E731

    def call(topk):
        keep = [i64(0, 1), i64(0), i64(4), i64(0, 4), torch.arange(4).cuda(), torch.zeros(4 * 512 * 8, dtype=torch.int64).cuda()]
        off, lo, hi, win, part, z = (K.ptr(t) for t in keep)
        out = [z + 8192 * k for k in range(8)]
        if entry == "counts":
            args = (1, off, lo, hi, win, z, 4, part, 1, topk, 1, 2 * topk, *out[1:4], out[4], out[5], out[6], out[7], out[7])
            f = L.vk_select_topk
        else:
            args = (1, off, lo, hi, win, z, z, z, z, z, z, topk, 1, part, 2 * topk, *out[1:4], out[4], out[5], out[6], out[7])
            f = L.vk_select_hits
        return lambda: keep and f(*args, K.stream())
    assert not _pair([call(40), call(500)], 3000)
