"""Kernels that are sent to the device while the one in front of them still runs: each sees all that was written before it."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows, batch, pages", [(1, 1, 3), (4, 4, 40), (16, 5, 1), (16, 300, 30)])
def test_chains_equal_synchronised_ones(cuda_device, dtype, rows, batch, pages):
    # small and large kernels in turn, in front of and behind each other and behind plain launches, over buffers that the allocator
    # hands out again at once: the bits are those of a run that waits for the device after every call
    from kinetics_b200 import ops
    g = torch.Generator().manual_seed(rows + batch)
    dev, Hq, Hkv, D, cols = cuda_device, 4, 1, 128, 512
    put = lambda *s: torch.randn(*s, generator=g).to(dtype).to(dev)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    w, wn, wq = put(cols, cols) * cols ** -0.5, put(cols), put(D)
    x0, hidden0, cache0 = put(rows, cols), put(batch, (Hq + 2 * Hkv) * D), put(batch * pages, 2, 16, Hkv, D)
    indices, indptr, last = i32(list(range(batch * pages))), i32([b * pages for b in range(batch + 1)]), i32([5] * batch)
    status = ops.new_status(dev)

    def chain(cache, wait):
        x, hidden = x0, hidden0
        summaries = torch.zeros(batch, Hkv, pages, D, device=dev, dtype=dtype)
        ops.build_summaries(cache, summaries, indices, indptr, last)
        kept = []
        for step in range(12):
            x, n = ops.add_rmsnorm(x, x0, wn, 1e-6); wait()
            n = ops.linear_rows(n, w); wait()
            x = ops.silu_mul(n, x); wait()
            x = x.clone() if step % 3 == 1 else x; wait()
            q, k, v = ops.qkv_norm(hidden, wq, wq, 1e-6, Hq, Hkv); wait()
            ops.append_kv(k, v, cache, summaries, indices, indptr, last, status=status); wait()
            sel = ops.select_pages(q, summaries, indices, indptr, last, 4, batch * pages, status=status); wait()
            sel = sel[0] if isinstance(sel, tuple) else sel
            o = ops.sparse_decode(q, cache, sel, indptr, last, status=status); wait()
            o = o + ops.dense_decode(q, cache, indices, indptr, last, pages, status=status); wait()
            hidden = torch.cat((o.reshape(batch, -1), hidden[:, Hq * D:]), dim=1); wait()
            kept += [x, o]
        return kept + [cache, summaries]
    want = chain(cache0.clone(), torch.cuda.synchronize)
    for _ in range(3):
        got = chain(cache0.clone(), lambda: None)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    side, graph, cache = torch.cuda.Stream(), torch.cuda.CUDAGraph(), cache0.clone()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain(cache, lambda: None)
    torch.cuda.current_stream().wait_stream(side)
    with torch.cuda.graph(graph):
        got = chain(cache, lambda: None)
    for _ in range(3):
        cache.copy_(cache0)
        graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    ops.raise_on_status(status)


def test_a_launch_that_fails_leaves_no_error_behind(cuda_device):
    # a capture that was ended by a forbidden call refuses launches on its stream; the next operation, elsewhere, is none the wiser
    from kinetics_b200 import _lib, ops
    lib, runtime, stream = _lib.load(), ctypes.CDLL("libcudart.so.12"), torch.cuda.Stream()
    x, w = torch.randn(4, 64, device=cuda_device), torch.randn(32, 64, device=cuda_device)
    out, on = torch.empty(4, 32, device=cuda_device), ctypes.c_void_p(stream.cuda_stream)
    torch.cuda.synchronize()
    assert runtime.cudaStreamBeginCapture(on, 2) == 0
    assert runtime.cudaStreamSynchronize(on) != 0
    rc = lib.ktk_linear_rows(x.data_ptr(), w.data_ptr(), None, None, None, out.data_ptr(), 4, 32, 64, _lib.KTK_F32, on)
    text, graph = lib.ktk_last_error(), ctypes.c_void_p()
    assert runtime.cudaStreamEndCapture(on, ctypes.byref(graph)) != 0
    runtime.cudaGetLastError()                               # the test's own calls
    assert rc != 0 and b"CUDA error" in text
    torch.testing.assert_close(ops.rmsnorm(x, torch.ones(64, device=cuda_device), 1e-6),
                               torch.nn.functional.rms_norm(x, (64,), eps=1e-6), rtol=1e-5, atol=1e-5)
