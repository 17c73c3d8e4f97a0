"""The prompt-sized products take their scratch from a pool of the device: a stream capture may hold the first such call that a process makes, and calls
from several threads on streams of their own do not meet in it.  Results are compared bit for bit with eager calls on one stream."""
import ctypes as C
import os
import subprocess
import sys
import threading

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

pytestmark = pytest.mark.gpu

BF16, Q4_K, Q6_K = 30, 12, 14
ROWS = {"linear": 40, "mlp": 18, "fp8": 17, "experts": 48}      # about the smallest batches of these paths at the sizes below


def _call(kind, seed=1, rows=None):
    """(input, output, call): a loaded handle's forward on the current stream; nothing of `kind` has run yet"""
    from ktransformers_b200 import native
    from ktransformers_b200.util.synth import synth_blocks
    lib, T, h = native.lib(), rows or ROWS[kind], C.c_void_p()
    stream = lambda: torch.cuda.current_stream().cuda_stream
    K, R, E, k = 1024, 512, 4, 2
    x, y = torch.zeros((T, K), dtype=torch.bfloat16, device="cuda"), torch.zeros((T, R if kind in ("linear", "fp8") else K), dtype=torch.bfloat16, device="cuda")
    if kind == "linear":
        keep = synth_blocks(Q4_K, R * K, "cuda", seed)
        native.check(lib.ktb200_linear_create(K, R, keep.data_ptr(), Q4_K, BF16, T, 0, C.byref(h)))
        native.check(lib.ktb200_linear_load_weights(h, stream()))
        run = lambda: native.check(lib.ktb200_linear_forward(h, T, x.data_ptr(), y.data_ptr(), None, None, stream()))
    elif kind == "mlp":
        keep = [synth_blocks(t, R * K, "cuda", seed + i) for i, t in enumerate((Q4_K, Q4_K, Q6_K))]
        native.check(lib.ktb200_mlp_create(K, R, *[t.data_ptr() for t in keep], Q4_K, Q4_K, Q6_K, BF16, T, 0, C.byref(h)))
        native.check(lib.ktb200_mlp_load_weights(h, stream()))
        run = lambda: native.check(lib.ktb200_mlp_forward(h, T, x.data_ptr(), y.data_ptr(), 0, None, stream()))
    elif kind == "fp8":
        g = torch.Generator(device="cuda").manual_seed(seed)
        keep = (torch.randn((R, K), generator=g, device="cuda") * 50).to(torch.float8_e4m3fn), torch.rand((R // 128, K // 128), generator=g, device="cuda")
        native.check(lib.ktb200_fp8_linear_create(K, R, keep[0].data_ptr(), keep[1].data_ptr(), BF16, 0, C.byref(h)))
        run = lambda: native.check(lib.ktb200_fp8_linear_forward(h, T, x.data_ptr(), y.data_ptr(), None, stream()))
    else:
        w = [synth_blocks(t, E * R * K, "cuda", seed + i) for i, t in enumerate((Q4_K, Q4_K, Q6_K))]
        cfg = native.MoeConfig(E, k, K, R, 64, 10, T, 1, *[t.data_ptr() for t in w], Q4_K, Q4_K, Q6_K, BF16, 0)
        native.check(lib.ktb200_moe_create(C.byref(cfg), 0, C.byref(h)))
        native.check(lib.ktb200_moe_load_weights(h, stream()))
        ids = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).cuda()
        wt = torch.rand((T, k), device="cuda")
        keep = w, ids, wt
        run = lambda: native.check(lib.ktb200_moe_forward(h, T, k, ids.data_ptr(), wt.data_ptr(), x.data_ptr(), y.data_ptr(), None, stream()))
    run.keep = keep
    return x, y, run


def _inputs(x, seed):
    return torch.randn(x.shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(x.dtype)


def _captured_first(kind):
    x, y, run = _call(kind)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    got = []
    for seed in (1, 2, 1):
        x.copy_(_inputs(x, seed))
        graph.replay()
        got.append(y.clone())
    for seed, g in zip((1, 2, 1), got):
        x.copy_(_inputs(x, seed))
        y.zero_()
        run()
        assert torch.isfinite(y.float()).all() and y.float().abs().max() > 0
        assert torch.equal(y, g), seed


@pytest.mark.parametrize("kind", list(ROWS))
def test_the_first_call_of_a_process_may_be_captured(kind):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), kind], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_two_threads_on_two_streams():
    jobs = [(_call(kind, seed, rows), seed) for seed, (kind, rows) in enumerate([("linear", 300), ("experts", 200), ("mlp", 150), ("fp8", 400)] * 2)]
    for (x, y, run), seed in jobs:
        x.copy_(_inputs(x, seed))
        run()
    torch.cuda.synchronize()
    want = [job[0][1].clone() for job in jobs]
    failed = []

    def work(part):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(20):
                    for i in part:
                        jobs[i][0][1].zero_()
                        jobs[i][0][2]()
                        if not torch.equal(jobs[i][0][1], want[i]):
                            failed.append(i)
        except Exception as e:
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(part,)) for part in (range(0, 4), range(4, 8))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


# decode sizes: one kernel with two sizes of shared memory, a thread each.  Linears of one row (two CTAs an SM) and of six (one), MLPs through both row kernels
@pytest.mark.parametrize("kind,rows,sizes", [("linear", 1, [(16384, 512), (1024, 512)]), ("linear", 6, [(14336, 512), (2048, 512)]), ("mlp", 1, [(16384, 512), (4096, 256)]), ("mlp", 4, [(8192, 2048), (4096, 512)])])
def test_two_threads_with_one_kernel_at_two_sizes(kind, rows, sizes):
    from ktransformers_b200 import native
    from ktransformers_b200.util.synth import synth_blocks
    lib, jobs, failed = native.lib(), [], []
    for K, R in sizes:
        h = C.c_void_p()
        keep = [synth_blocks(t, R * K, "cuda", 1 + i) for i, t in enumerate((Q4_K, Q4_K, Q6_K))]
        if kind == "linear":
            native.check(lib.ktb200_linear_create(K, R, keep[0].data_ptr(), Q4_K, BF16, rows, 0, C.byref(h)))
            native.check(lib.ktb200_linear_load_weights(h, torch.cuda.current_stream().cuda_stream))
        else:
            native.check(lib.ktb200_mlp_create(K, R, *[t.data_ptr() for t in keep], Q4_K, Q4_K, Q6_K, BF16, rows, 0, C.byref(h)))
            native.check(lib.ktb200_mlp_load_weights(h, torch.cuda.current_stream().cuda_stream))
        x = _inputs(torch.empty((rows, K), dtype=torch.bfloat16, device="cuda"), K)
        y, want = (torch.zeros((rows, R if kind == "linear" else K), dtype=torch.bfloat16, device="cuda") for _ in range(2))

        def call(y, stream, h=h, x=x):
            if kind == "linear":
                return lib.ktb200_linear_forward(h, rows, x.data_ptr(), y.data_ptr(), None, None, stream)
            return lib.ktb200_mlp_forward(h, rows, x.data_ptr(), y.data_ptr(), 0, None, stream)

        native.check(call(want, torch.cuda.current_stream().cuda_stream))
        jobs.append((call, y, want, keep))
    torch.cuda.synchronize()

    def work(call, y, want, keep):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                stream = torch.cuda.current_stream().cuda_stream
                for i in range(3000):
                    native.check(call(y, stream))
                if not torch.equal(y, want):
                    failed.append("other bits")
        except Exception as e:
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


if __name__ == "__main__":
    _captured_first(sys.argv[1])
