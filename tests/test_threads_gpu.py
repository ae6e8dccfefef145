"""Operators called from several Python threads: a launch does not stop the other threads, and calls that share a
stream, and with it the scratch buffer, do not mix their kernels."""
import gc
import sys
import threading

import pytest
import torch

from conftest import make_activation, make_weight

pytestmark = pytest.mark.gpu


def _linear(M, N, K, seed):
    import sglang_b200 as S

    wq, ws = make_weight(N, K, seed)
    x, wq, ws = make_activation(M, K, seed + 1).cuda(), wq.cuda(), ws.cuda()
    return lambda: S.w8a8_block_fp8_linear(x, wq, [128, 128], ws)


def _native_calls():
    """One call of each function of the native host path, by its name there."""
    import sglang_b200 as S
    from sglang_b200 import _native as N

    x = make_activation(32, 512, 1).cuda()
    wq, ws = (t.cuda() for t in make_weight(256, 512, 2))
    q, s = S.per_token_group_quant_fp8(x, 128)
    qp, sp = S.per_token_group_quant_fp8(x, 128, column_major_scales=True, scale_tma_aligned=True, scale_ue8m0=True)
    wsp = torch.full((1, 256), 0x7F7F7F7F, dtype=torch.int32, device="cuda").t()
    logits = torch.randn(32, 8, generator=torch.Generator().manual_seed(5)).cuda()
    w1 = torch.zeros(8, 256, 512, device="cuda").to(torch.float8_e4m3fn)
    w2 = torch.zeros(8, 512, 128, device="cuda").to(torch.float8_e4m3fn)
    w1_s, w2_s = torch.ones(8, 2, 4, device="cuda"), torch.ones(8, 4, 1, device="cuda")
    tw, ti = S.fused_topk(x, logits, 2, True)
    args = {
        "linear": (x, wq, ws),
        "quant": (x, 128, False, False, False, 0, 1e-10),
        "matmul": (q, wq, s, ws, N.BF16),
        "matmul_ue8m0": (qp, wq, sp, wsp, N.BF16),
        "route": (logits, None, 2, 0, 0, 0, 0, True, 1.0),
        "experts": (x, w1, w2, tw, ti, w1_s, w2_s, False, False, False, None),
    }
    return {name: (getattr(N.host, name), a) for name, a in args.items()}


@pytest.mark.parametrize("name", ["linear", "quant", "matmul", "matmul_ue8m0", "route", "experts"])
def test_launches_give_the_interpreter_lock_back(name):
    """Another thread gets its turn while calls wait for room in the launch queue behind 0.2 s of work. The interpreter
    takes the lock from nobody here (its switch interval is far longer than the test), so that thread can only run when
    a call gives it back. Results are kept: freeing one may give it back too."""
    call, args = _native_calls()[name]
    assert call(*args) is not None
    torch.cuda.synchronize()
    go, ran, results = threading.Event(), [], []
    other = threading.Thread(target=lambda: (go.wait(), ran.append(1)))
    other.start()
    interval = sys.getswitchinterval()
    sys.setswitchinterval(100.0)
    gc.disable()
    try:
        torch.cuda._sleep(400_000_000)
        go.set()
        for _ in range(3000):
            results.append(call(*args))
            if ran:
                break
        assert ran
    finally:
        gc.enable()
        sys.setswitchinterval(interval)
        other.join()
        torch.cuda.synchronize()


def test_two_threads_on_one_stream():
    """Quantised activations and K-split partial sums of one call lie in the scratch that the next call on the stream
    reuses: with two threads launching to the same stream every result is still its own (bit for bit)."""
    calls = [_linear(200, 1024, 2048, 10), _linear(17, 512, 4096, 20), _linear(64, 2048, 1024, 30)]
    want = [c().clone() for c in calls]
    stream = torch.cuda.current_stream()
    wrong = []

    def work(k):
        with torch.cuda.stream(stream):
            for _ in range(300):
                if not torch.equal(calls[k](), want[k]):
                    wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("entry", ["b200_w8a8_block_fp8_gemm", "b200_moe_align_block_size", "b200_fused_experts_fp8",
                                   "b200_fused_experts_fp8_scatter", "b200_masked_experts_fp8"])
def test_general_paths_keep_the_scratch_to_themselves(entry, monkeypatch):
    """The Python wrappers launch through ctypes, which lets other threads run: while one of their calls is under way,
    the stream's scratch is not lent to another thread."""
    import sglang_b200 as S
    from sglang_b200 import _native as N
    from sglang_b200.fp8_kernel import _workspace
    from sglang_b200.fused_moe import fused_experts_impl, fused_experts_scatter

    x = make_activation(300, 256, 1).cuda()
    q, s = S.per_token_group_quant_fp8(x, 128)
    wq, ws = (t.cuda() for t in make_weight(256, 256, 2))
    w1 = torch.zeros(8, 256, 256, device="cuda").to(torch.float8_e4m3fn)
    w2 = torch.zeros(8, 256, 128, device="cuda").to(torch.float8_e4m3fn)
    w1_s, w2_s = torch.ones(8, 2, 2, device="cuda"), torch.ones(8, 2, 1, device="cuda")
    tw = torch.ones(300, 4, device="cuda")
    ti = (torch.arange(1200, device="cuda", dtype=torch.int32) % 8).view(300, 4)
    rows = torch.zeros(1200, 256, dtype=torch.bfloat16, device="cuda")
    dest = (N.c_void_p * 1)(rows.data_ptr())
    calls = {
        # a 3-D input takes the general path; 64 rows of K = 2048 would split K
        "b200_w8a8_block_fp8_gemm": lambda: S.w8a8_block_fp8_matmul(q.view(1, 300, 256), wq, s.view(1, 300, 2), ws, [128, 128]),
        "b200_moe_align_block_size": lambda: S.moe_align_block_size(ti, 16, 8),
        "b200_fused_experts_fp8": lambda: fused_experts_impl(q, w1, w2, tw, ti, w1_s, w2_s, inplace=False,
                                                             hidden_states_scale=s, output_dtype=torch.bfloat16),
        "b200_fused_experts_fp8_scatter": lambda: fused_experts_scatter(q, s, w1, w2, tw, ti, w1_s, w2_s, dest, 1200,
                                                                        torch.bfloat16),
        "b200_masked_experts_fp8": lambda: S.masked_fused_experts(
            q[:256].repeat(8, 1).view(8, 256, 256), s[:256].repeat(8, 1).view(8, 256, 2), w1, w1_s, w2, w2_s,
            torch.full((8,), 5, dtype=torch.int32, device="cuda")),
    }
    lib, device = N.load(), torch.device("cuda", torch.cuda.current_device())
    real, waited = getattr(lib, entry), []

    def probe(*args):
        thread = threading.Thread(target=_workspace, args=(device, 1))
        thread.start()
        thread.join(0.1)
        waited.append((thread, thread.is_alive()))
        return real(*args)

    with N.tuning(gemm_splitk=2):
        monkeypatch.setattr(lib, entry, probe)
        calls[entry]()
    (thread, alive), = waited
    thread.join(10)
    assert alive and not thread.is_alive()
    assert N.read_device_status() == 0
