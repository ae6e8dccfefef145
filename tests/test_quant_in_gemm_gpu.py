"""The decode kernel that quantises its own input against quantiser and GEMM on their own: the same bytes, scales, K splits and
order of the sums, so the same bits at every shape that takes it."""
import ctypes

import pytest
import torch

from conftest import make_activation

pytestmark = pytest.mark.gpu


def _weight(N, K, seed):
    """Weight bytes and scales that keep the spread of the activations about one."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.empty(N, K, dtype=torch.float8_e4m3fn, device="cuda")
    for rows in torch.arange(N).split(4096):  # a part at a time: the largest weight is half a gigabyte
        w[rows[0] : rows[-1] + 1] = ((torch.rand(len(rows), K, device="cuda", generator=g) - 0.5) * 400).to(w.dtype)
    s = (torch.rand((N + 127) // 128, K // 128, device="cuda", generator=g) + 0.5) / (115 * K**0.5)
    return w, s


def _same_bits(a, b):
    return torch.equal(a.view(torch.int16), b.view(torch.int16))


def _takes_it(M, N, K):
    """Both routes, checked: the kernel with the quantiser (which the plan takes where it is the faster one, here everywhere), and
    the decode kernel with the same splits behind a quantiser."""
    from sglang_b200 import _native as N_

    with N_.tuning(linear_decode_fused=2):
        fused = N_.plan_dense("linear", M, N, K)
    with N_.tuning(linear_decode_fused=0):
        apart = N_.plan_dense("linear", M, N, K)
    assert fused.kernel == "skinny_quant" and apart == fused._replace(kernel="skinny")


def _fused():
    from sglang_b200 import _native as N_

    return N_.tuning(linear_decode_fused=2)


# unsplit with one wave and with two, the largest scale table (64 K blocks a CTA), clusters of 2 to 8, a short last split,
# ragged columns, fewer K blocks than four groups of lanes have in flight
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("N,K", [(6144, 4096), (28672, 4096), (4096, 14336), (4096, 4096), (5000, 4096), (38400, 512), (57344, 8192)])
def test_same_bits_as_quantiser_and_gemm(M, N, K, dtype):
    import sglang_b200 as S
    from sglang_b200 import _native as N_

    _takes_it(M, N, K)
    x, (w, s) = make_activation(M, K, M + K, dtype=dtype).cuda(), _weight(N, K, N + K)
    with _fused():
        out = S.w8a8_block_fp8_linear(x, w, [128, 128], s)
    with N_.tuning(linear_decode_fused=0):
        apart = S.w8a8_block_fp8_linear(x, w, [128, 128], s)
    assert N_.read_device_status() == 0
    assert out.dtype == dtype and _same_bits(out, apart) and bool(out.float().abs().max() > 0)


# small weights: clusters of 5 to 8, a last split of one K block, one K block in all, fewer columns than a tile
@pytest.mark.parametrize("M,N,K", [(4, 136, 8320), (8, 136, 8320), (5, 1280, 8192), (8, 1280, 8192), (8, 520, 16384), (8, 8, 128),
                                   (3, 1032, 384), (7, 2048, 2176)])
def test_same_bits_with_small_weights(M, N, K):
    test_same_bits_as_quantiser_and_gemm(M, N, K, torch.bfloat16)


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (8, 28672, 1024), (8, 1280, 8192)])
def test_input_written_right_before_the_call(M, N, K):
    """A copy kernel writes x, then the call, with nothing between: the kernel's CTAs start before the copy has finished."""
    import sglang_b200 as S
    from sglang_b200 import _native as N_

    _takes_it(M, N, K)
    w, s = _weight(N, K, 5)
    kept = [make_activation(M, K, i).cuda() for i in (1, 2)]
    want = [S.w8a8_block_fp8_linear(x, w, [128, 128], s) for x in kept]
    torch.cuda.synchronize()
    x, wrong = torch.empty_like(kept[0]), []
    with _fused():
        for i in range(40):
            x.copy_(kept[i % 2])
            wrong.append((S.w8a8_block_fp8_linear(x, w, [128, 128], s) != want[i % 2]).sum())
    assert int(torch.stack(wrong).sum()) == 0
    assert N_.read_device_status() == 0


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (8, 4096, 14336), (1, 1536, 4096)])
def test_one_kernel_needs_no_workspace(M, N, K):
    import sglang_b200 as S
    from sglang_b200 import _native as N_

    assert N_.plan_dense("linear", M, N, K).kernel.endswith("quant")
    x, (w, s) = make_activation(M, K, 6).cuda(), _weight(N, K, 7)
    out = torch.empty(M, N, dtype=x.dtype, device="cuda")
    st = N_.load().b200_w8a8_block_fp8_linear(x.data_ptr(), N_.BF16, w.data_ptr(), s.data_ptr(), out.data_ptr(), M, N, K, None, 0,
                                              N_.current_stream())
    N_.check(st, "linear")
    assert _same_bits(out, S.w8a8_block_fp8_linear(x, w, [128, 128], s))
    assert N_.read_device_status() == 0


@pytest.mark.parametrize("M", [1, 8])
def test_chain_through_two_buffers(M):
    """Linears that read what the one before has written and overwrite what it has read: each starts while the one before, and
    perhaps the one before that, still runs."""
    from sglang_b200 import _native as N_

    n = 4096
    _takes_it(M, n, n)
    lib, weights = N_.load(), [_weight(n, n, 10 + i) for i in range(3)]
    first = make_activation(M, n, 9).cuda()
    need = lib.b200_w8a8_block_fp8_linear_workspace_bytes(M, n, n)
    scratch = torch.empty(need, dtype=torch.uint8, device="cuda")

    def chain(steps, pause):
        bufs, seen = [first.clone(), torch.empty_like(first)], []
        for i in range(steps):
            w, s = weights[i % 3]
            src, dst = bufs[i % 2], bufs[(i + 1) % 2]
            N_.check(lib.b200_w8a8_block_fp8_linear(src.data_ptr(), N_.BF16, w.data_ptr(), s.data_ptr(), dst.data_ptr(), M, n, n,
                                                    scratch.data_ptr(), ctypes.c_size_t(need), N_.current_stream()), "linear")
            if pause:
                torch.cuda.synchronize()
        return bufs[steps % 2]

    for steps in (2, 3, 10, 31):
        with _fused():
            got = chain(steps, pause=False)
        with N_.tuning(linear_decode_fused=0):
            want = chain(steps, pause=True)
        assert _same_bits(got, want), steps
        assert bool(torch.isfinite(got).all()) and bool(got.float().abs().max() > 0)
    assert N_.read_device_status() == 0
