"""Weights written on the stream right before the call that reads them. The weight-streaming kernels start before the
kernels ahead of them have finished; the weights are ordered like every other operand all the same."""
import pytest
import torch

from conftest import make_activation

pytestmark = pytest.mark.gpu
FP8 = torch.float8_e4m3fn


def _bytes(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return ((torch.rand(shape, device="cuda", generator=g) - 0.5) * 400).to(FP8)


# one launch; decode kernel with its K splits in a cluster and without; token tiles of 64; a prefill tile
@pytest.mark.parametrize("M,N,K", [(1, 1536, 4096), (1, 4096, 4096), (17, 28672, 1024), (61, 3584, 4096), (300, 1024, 1024)])
def test_linear_after_a_weight_update(M, N, K):
    import sglang_b200 as S
    from sglang_b200 import _native as N_

    x = make_activation(M, K, 3).cuda()
    ws = torch.rand((N + 127) // 128, K // 128, device="cuda") * 1e-3
    kept = [_bytes((N, K), s) for s in (1, 2)]
    want = [S.w8a8_block_fp8_linear(x, w, [128, 128], ws) for w in kept]
    torch.cuda.synchronize()
    w, wrong = torch.empty_like(kept[0]), []
    for i in range(40):  # a copy kernel, then the call, with nothing between
        w.view(torch.int64).copy_(kept[i % 2].view(torch.int64))
        wrong.append((S.w8a8_block_fp8_linear(x, w, [128, 128], ws) != want[i % 2]).sum())
    assert int(torch.stack(wrong).sum()) == 0
    assert N_.read_device_status() == 0


def test_matmul_of_just_quantised_weights():
    """The bytes of the stand-alone quantiser as the next GEMM's weights."""
    import sglang_b200 as S

    N, K = 4096, 2048
    q, s = S.per_token_group_quant_fp8(make_activation(8, K, 4).cuda(), 128)
    ws = torch.rand(N // 128, K // 128, device="cuda") * 1e-3
    raw = [torch.randn(N, K, device="cuda").bfloat16() for _ in range(2)]
    want = [S.w8a8_block_fp8_matmul(q, S.per_token_group_quant_fp8(r, 128)[0], s, ws, [128, 128]) for r in raw]
    torch.cuda.synchronize()
    wrong = []
    for i in range(40):
        w, _ = S.per_token_group_quant_fp8(raw[i % 2], 128)
        wrong.append((S.w8a8_block_fp8_matmul(q, w, s, ws, [128, 128]) != want[i % 2]).sum())
    assert int(torch.stack(wrong).sum()) == 0


@pytest.mark.parametrize("T,E,topk", [(1, 16, 2), (40, 8, 2)])
def test_experts_after_a_weight_update(T, E, topk):
    import sglang_b200 as S
    from sglang_b200 import _native as N

    H, I = 1024, 512
    x = make_activation(T, H, 5).cuda()
    tw, ti = S.fused_topk(x, torch.randn(T, E, device="cuda"), topk, True)
    w1_s, w2_s = torch.rand(E, 2 * I // 128, H // 128, device="cuda") * 1e-3, torch.rand(E, H // 128, I // 128, device="cuda") * 1e-3
    kept = [(_bytes((E, 2 * I, H), s), _bytes((E, H, I), s + 10)) for s in (1, 2)]

    def call(w1, w2):
        return S.fused_experts(x, w1, w2, S.StandardTopKOutput(tw, ti, None), S.MoeRunnerConfig(inplace=False), use_fp8_w8a8=True,
                               w1_scale=w1_s, w2_scale=w2_s, block_shape=[128, 128])

    want = [call(*k) for k in kept]
    torch.cuda.synchronize()
    w1, w2, wrong = torch.empty_like(kept[0][0]), torch.empty_like(kept[0][1]), []
    for i in range(40):
        w1.view(torch.int64).copy_(kept[i % 2][0].view(torch.int64))
        w2.view(torch.int64).copy_(kept[i % 2][1].view(torch.int64))
        wrong.append((call(w1, w2) != want[i % 2]).sum())
    assert int(torch.stack(wrong).sum()) == 0
    assert N.read_device_status() == 0


def test_layers_back_to_back_on_the_shared_scratch():
    """Several layers in a row without a synchronisation, of every kind and size class, each with its own weights: the
    kernels of one layer start while those of the last one drain, and all pass their intermediates through the same
    scratch. Every output equals the one of the same layer run alone."""
    import sglang_b200 as S
    from sglang_b200 import _native as N

    calls = []
    for i, (M, N_, K) in enumerate([(1, 512, 1024), (3, 4096, 1024), (64, 1024, 2048), (200, 512, 4096), (17, 2048, 1024),
                                    (1000, 512, 512)]):
        x, w = make_activation(M, K, 20 + i).cuda(), _bytes((N_, K), 30 + i)
        ws = torch.rand(N_ // 128, K // 128, device="cuda") * 1e-3
        calls.append(lambda x=x, w=w, ws=ws: S.w8a8_block_fp8_linear(x, w, [128, 128], ws))
    for i, (T, E, topk) in enumerate([(1, 16, 4), (30, 16, 4), (300, 16, 4), (700, 8, 2), (2, 8, 2)]):
        H, I = 512, 256
        x = make_activation(T, H, 50 + i).cuda()
        w1, w2 = _bytes((E, 2 * I, H), 60 + i), _bytes((E, H, I), 70 + i)
        s1, s2 = torch.rand(E, 2 * I // 128, H // 128, device="cuda") * 1e-3, torch.rand(E, H // 128, I // 128, device="cuda") * 1e-3
        logits = torch.randn(T, E, device="cuda")

        def layer(x=x, w1=w1, w2=w2, s1=s1, s2=s2, logits=logits, topk=topk):
            tw, ti = S.fused_topk(x, logits, topk, True)
            return S.fused_experts(x, w1, w2, S.StandardTopKOutput(tw, ti, None), S.MoeRunnerConfig(inplace=False),
                                   use_fp8_w8a8=True, w1_scale=s1, w2_scale=s2, block_shape=[128, 128])

        calls.insert(2 * i, layer)
    alone = []
    for c in calls:
        alone.append(c().clone())
        torch.cuda.synchronize()
    wrong = []
    for r in range(20):
        order = torch.randperm(len(calls), generator=torch.Generator().manual_seed(r)).tolist()
        outs = [calls[k]() for k in order]
        wrong += [(o != alone[k]).sum() for o, k in zip(outs, order)]
    assert int(torch.stack(wrong).sum()) == 0
    assert N.read_device_status() == 0
