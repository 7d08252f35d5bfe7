"""How the weight-streaming GEMM cuts a problem.  The K split decides the order of the sums, so a plan follows from the sizes and from
nothing that differs from one GPU, thread or process to the next."""
import ctypes
import os
import random
import threading

import pytest
import torch

from ooverlap_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def plan(M, N, K, pair=0, splits=0, b_static=0, one_block=0):
    out = (ctypes.c_int * 6)()
    assert _lib.lib().oob_test_gemm_cluster_plan(M, N, K, pair, splits, b_static, one_block, out) == 0
    return tuple(out)[:5]


def leaves_l2_first(M, N, K, b_static=0):
    out = (ctypes.c_int * 6)()
    assert _lib.lib().oob_test_gemm_cluster_plan(M, N, K, 0, 0, b_static, 0, out) == 0
    return bool(out[5])


def shapes(n, seed):
    rng = random.Random(seed)
    return [(int(2 ** rng.uniform(0, 12)), 8 * rng.randint(8, 1024), 8 * rng.randint(8, 1024)) for _ in range(n)]


# Token blocks, tokens of a block, pairs, K splits, CTAs an SM: shapes whose clusters come close to what a GPU runs at once, where one
# cluster fewer has another K split.
PINNED = {(154, 5568, 2584): (1, 160, 1, 3, 1), (116, 1024, 5624): (1, 128, 0, 8, 1), (512, 1280, 8192): (3, 176, 1, 3, 1),
          (256, 4096, 4096): (2, 128, 0, 2, 1), (100, 2048, 2048): (4, 32, 0, 2, 1), (16, 7168, 8192): (1, 16, 0, 2, 1)}


def check_pinned():
    for shape, want in PINNED.items():
        assert plan(*shape) == want, shape


def test_pinned_plans_without_a_device():
    check_pinned()


@pytest.mark.gpu
def test_pinned_plans_on_a_device():
    torch.zeros(1, device="cuda")
    check_pinned()


def test_planning_asks_no_device():
    with open(os.path.join(ROOT, "csrc", "gemm", "gemm_cluster.cu")) as f:
        assert "cudaOccupancy" not in f.read().replace("(cudaOccupancyMaxActiveClusters)", "")


def test_threads_agree():
    want = [plan(*s) for s in shapes(400, 1)]
    got = {}

    def other(i):
        order = list(enumerate(shapes(400, 1)))
        random.Random(i).shuffle(order)
        got[i] = [p for _, p in sorted((j, plan(*s)) for j, s in order)]

    threads = [threading.Thread(target=other, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(got[i] == want for i in range(3))


def test_plans_are_sound():
    for M, N, K in shapes(600, 2):
        blocks, tokens, pair, S, per_sm = plan(M, N, K)
        assert tokens % 16 == 0 and blocks * tokens >= M > (blocks - 1) * tokens and tokens <= 384
        assert 1 <= S * (2 if pair else 1) <= 8 and 1 <= per_sm <= 4
        if M <= 128:
            assert plan(M, N, K, one_block=1)[0] == 1
        assert plan(M, N, K, splits=1)[3] == 1


def test_weights_that_stay_in_l2_are_kept_there():
    """A weight of up to some 70 MB that is used again and again is in L2 the next time, whether it is promised not to be written or not; only
    the caller knows that it is one of many."""
    for mb, alone in ((4, False), (16, False), (48, False), (72, False), (79, False), (81, True), (200, True)):
        N = mb * (1 << 20) // (2 * 4096)
        assert leaves_l2_first(16, N, 4096) == alone and leaves_l2_first(16, N, 4096, 1) == alone, mb
        assert leaves_l2_first(16, N, 4096, 2) == (mb >= 8), mb
    assert not leaves_l2_first(1000, 16384, 4096)  # several token blocks read it


def test_a_model_says_that_its_weights_exceed_l2():
    from ooverlap_b200.models import llama
    from ooverlap_b200.ops.gemm import _scope
    m = llama.LlamaTP(llama.TINY, None, dtype=torch.bfloat16, device=torch.device("cpu"), max_batch=8, max_len=16)
    assert m.weight_bytes == sum(w.numel() * 2 for layer in m.layers for k, w in layer.items() if k.startswith("w")) + 2 * m.lm_head.numel()
    seen = []
    m._forward = lambda *a: seen.append(_scope.static_b)
    for mb, rows, want in ((8, 8, 1), (95, 8, 1), (96, 8, 2), (100, 1, 1), (128, 1, 2)):
        m.weight_bytes = mb << 20
        m.forward(torch.zeros(rows, 1, dtype=torch.long), 0)
        assert seen.pop() == want and not _scope.static_b


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [_lib.F16, _lib.BF16])
@pytest.mark.parametrize("epilogue", [0, 1, 2, 3])
def test_no_kernel_spills_its_sums(epilogue, dtype):
    """Loads of a turn wait for each other where a thread has too few registers for its sums.  (The SwiGLU kernels have 32 bytes of arrays that are
    indexed.)"""
    torch.zeros(1, device="cuda")
    assert _lib.lib().oob_test_gemm_cluster_local_bytes(epilogue, dtype) == (32 if epilogue == 1 else 0)
