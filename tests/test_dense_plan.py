"""The plan of the dense GEMMs and the linear layer (host arithmetic, no GPU)."""
import subprocess
import sys

from conftest import ROOT


def _plan(*a, **k):
    from sglang_b200 import _native as N

    return N.plan_dense(*a, **k)


def test_every_number_of_sms_has_a_plan():
    """Partitions of a GPU: down to one SM, sixteen among them, for sizes that reach every kernel. In a process of its own: an
    integer division by zero ends it."""
    code = """
from sglang_b200 import _native as N
for sms in range(1, 149):
    for M, n, k in [(1, 1536, 4096), (8, 4096, 4096), (33, 512, 1024), (64, 256, 8192), (100, 2048, 7168), (203, 4096, 4096),
                    (300, 200, 8192), (1027, 7168, 8192), (3000, 4096, 14336)]:
        for entry in ("gemm", "fanout", "linear", "packed"):
            p = N.plan_dense(entry, M, n, k, sms)
            assert 1 <= p.splits <= k // 128, (entry, M, n, k, sms, p)
            if sms < 2:
                assert p.kernel != "wide" or p.tile_n == 0, (entry, M, n, k, p)  # a CTA pair takes two SMs
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])


def test_few_tiles_split_k_on_a_partition():
    """Half of the part: four to eight tiles of a long K are not left to four CTAs or pairs (the whole part splits them in clusters)."""
    for sms in (36, 74, 132):
        for M, n, k in [(300, 512, 16384), (512, 256, 16384), (300, 512, 8192)]:
            p = _plan("gemm", M, n, k, sms)
            assert p.kernel == "wide" and p.splits > 1 and p.sum == "memory", (sms, M, n, k, p)
    assert _plan("gemm", 512, 256, 16384, 148).sum == "cluster"


def test_short_weights_of_some_rows_take_the_decode_kernel():
    """33 to 256 rows of weights with a short K, and a few wide ones: measured, the decode kernel is 4 to 27 % ahead of the pairs
    and single CTAs there (65 x 8192 x 512: 4.3 and 5.4 us)."""
    for n, k, rows in [(8192, 512, (65, 80, 96, 112, 128)), (16384, 1024, (40, 64)), (7168, 1024, (65, 96, 128, 144)),
                       (8192, 1024, (72, 100, 128)), (13560, 4736, (57,)), (10240, 8192, (65, 96)), (7144, 384, (134,)), (7616, 256, (79,))]:
        for m in rows:
            assert _plan("gemm", m, n, k, 148).kernel == "skinny", (m, n, k)
    # the other side of the line: 203 rows of a layer, and 61 rows on a rank of four
    assert _plan("gemm", 203, 4096, 4096, 148) == ("wide", 128, 2, "cluster")
    assert _plan("gemm", 203, 28672, 4096, 148).kernel == "wide"
    assert _plan("gemm", 61, 14336, 8192, 148).kernel == "stream"
    assert _plan("gemm", 957, 288, 256, 148) == ("wide", 128, 1, "none")


def test_packed_scales_take_the_decode_kernel_where_it_saves_the_unpacking():
    """The decode kernel reads packed words itself, every other kernel on fp32 scales waits for their unpacking. Measured:
    96 x 5120 x 1536 9.4 us block-scaled, 7.2 in the decode kernel; 204 x 336 x 1152 6.6 and 4.9; 64 x 16384 x 1024 8.9 on
    unpacked scales, 6.3."""
    for m, n, k in [(40, 16384, 1024), (64, 16384, 1024), (204, 336, 1152), (193, 312, 1024), (65, 5120, 1536), (80, 5120, 1536),
                    (96, 5120, 1536), (74, 264, 1024), (107, 816, 896), (57, 13560, 4736), (112, 1536, 7168)]:
        assert _plan("packed", m, n, k, 148).kernel == "skinny", (m, n, k)
    # CTA pairs where their start is paid back by K: 17.1 us against 17.9 of single CTAs; and where it is not
    for m in (100, 160, 203, 256):
        assert _plan("packed", m, 14336, 4096, 148).kernel == "block_scaled_pair", m
    assert _plan("packed", 400, 8192, 1024, 148).kernel == "block_scaled"
    assert _plan("packed", 3000, 4096, 14336, 148).kernel == "block_scaled_pair"
    assert _plan("packed", 203, 4096, 14336, 148).kernel == "wide"
    # large weights: unpacking is paid back by the weight-streaming kernel, 32 us against 35
    for m in (33, 48, 64):
        assert _plan("packed", m, 14336, 8192, 148).kernel == "stream", m


def test_packed_workspace_covers_either_plan():
    """Partials of the decode kernel, or scales and partials of the plan on unpacked ones."""
    from sglang_b200 import _native as N

    lib = N.load()
    for m in (1, 33, 64, 100, 144, 200, 256, 300):
        for n, k in [(4096, 1024), (1536, 7168), (5120, 1536), (16384, 1024), (264, 8192), (4096, 14336)]:
            have = lib.b200_w8a8_block_fp8_gemm_packed_workspace_bytes(m, n, k)
            p = _plan("packed", m, n, k)
            need = p.splits * m * n * 4 if p.sum == "memory" else 0
            if p.kernel.startswith("block_scaled"):
                assert have == 0
            else:
                scales = 0 if p.kernel == "skinny" else 4 * (m + -(-n // 128)) * -(-k // 128)
                assert have >= need + scales and have > 0, (m, n, k, p)


def test_fanout_is_planned_from_kernels_that_can_fan_out():
    """No sums in clusters, no weight streaming, and no kernel's time that the call does not run. Measured with the buffers on one
    GPU: 72 x 6144 x 4096 11.4 us in the decode kernel, 22.2 as the unsplit tile kernel that a plan for the streaming kernel ends in;
    320 x 2112 x 7168 34 unsplit, 17 in two splits."""
    for m, n, k in [(72, 6144, 4096), (112, 5120, 1536), (72, 8192, 3584), (128, 4096, 4096), (160, 3584, 4096), (65, 8192, 2048),
                    (128, 7168, 2048), (72, 4096, 4096), (160, 2560, 4096), (203, 2560, 4096)]:
        assert _plan("fanout", m, n, k, 148).kernel == "skinny", (m, n, k)
    for m, n, k in [(320, 2112, 7168), (384, 2112, 7168), (300, 4096, 14336), (158, 6912, 14336)]:
        assert _plan("fanout", m, n, k, 148) == ("wide", 128, 2, "memory"), (m, n, k)
    assert _plan("fanout", 1027, 8192, 3584, 148).kernel == "tile"
    for sms in (36, 148):
        for m in (1, 16, 33, 64, 100, 128, 200, 300, 512, 1027):
            for n, k in [(128, 8192), (200, 4096), (1024, 8192), (4096, 1792), (8192, 3584), (4096, 14336), (14336, 8192)]:
                p = _plan("fanout", m, n, k, sms)
                assert p.kernel in ("tile", "wide", "skinny") and p.sum != "cluster", p
                assert p.sum == "memory" or p.kernel == "tile", p  # the others write to the buffers in the reduction pass
                if p.kernel != "skinny":
                    assert (p.sum == "memory") == (p.splits > 1), p


def test_fanout_workspace_covers_its_plan():
    from sglang_b200 import _native as N

    lib = N.load()
    with N.tuning(gemm_2cta=1284, gemm_skinny=0):  # clusters asked for: a fan-out takes as many splits through memory
        assert lib.b200_w8a8_block_fp8_gemm_fanout_workspace_bytes(300, 1024, 4096) >= 4 * 300 * 1024 * 4
    for m in (1, 16, 33, 100, 256, 300, 700):
        for n, k in [(128, 8192), (200, 4096), (1024, 8192), (4096, 1792), (2112, 7168), (4096, 14336)]:
            p = _plan("fanout", m, n, k)
            need = p.splits * m * n * 4 if p.sum == "memory" else 0
            assert lib.b200_w8a8_block_fp8_gemm_fanout_workspace_bytes(m, n, k) >= need, (m, n, k, p)


def test_quantiser_in_the_decode_gemm_where_it_hides():
    """Measured against a quantiser of its own: ahead with at most one CTA per SM or two on nearly all and a long K, behind with
    a few SMs that have two CTAs (8 x 5120 x 5120 10.1 us and 9.0) or a short K (4 x 25416 x 1152 10.5 and 8.7)."""
    for m, n, k in [(1, 4096, 4096), (8, 4096, 4096), (8, 4096, 14336), (8, 28672, 4096), (1, 6144, 4096), (2, 6144, 4096), (8, 8192, 28672),
                    (8, 57344, 8192), (1, 8192, 3584), (8, 14336, 8192)]:
        assert _plan("linear", m, n, k, 148).kernel == "skinny_quant", (m, n, k)
    for m, n, k in [(8, 5120, 5120), (4, 5120, 5120), (2, 5120, 5120), (8, 4608, 7168), (8, 6144, 4096), (8, 8192, 3584), (4, 22336, 1152),
                    (1, 22400, 896), (4, 24576, 1536), (1, 32768, 512), (1, 16384, 1024), (9, 4096, 4096)]:
        assert _plan("linear", m, n, k, 148).kernel == "skinny", (m, n, k)


def test_clusters_have_the_splits_that_were_asked_for():
    """Two or four pairs, whatever K has: a split without K blocks adds zeros."""
    from sglang_b200 import _native as N

    for knob, splits in [(1282, 2), (1284, 4)]:
        for k in (128, 256, 384, 640, 4096):
            with N.tuning(gemm_2cta=knob, gemm_skinny=0):
                assert _plan("gemm", 200, 264, k, 148) == ("wide", 128, splits, "cluster"), (knob, k)


def test_narrow_outputs_are_not_split_for_nothing():
    """Fewer than 256 columns: a reduction pass costs 2 to 4 us, so 12 K blocks stay whole (502 x 192 x 1536 7.8 us, three splits
    11.5; packed 502 x 120 x 1536 8.6 in splits), 64 do not (300 x 128 x 8192 20.6 us whole, 9.2 in eight splits)."""
    for n in (64, 120, 128, 136, 192, 248):
        for m in (300, 502, 959):
            assert _plan("gemm", m, n, 1536, 148).splits == 1
            assert _plan("gemm", m, n, 8192, 148).splits >= 4
            p = _plan("packed", m, n, 1536, 148)
            assert p.kernel == "block_scaled" or p.splits == 1


def test_workspace_of_sums_in_clusters():
    """CTA pairs that sum their K splits in clusters write no partials; everything else is covered by the query."""
    from sglang_b200 import _native as N

    lib = N.load()
    for m, n, k in [(203, 4096, 4096), (203, 4096, 14336), (512, 1280, 8192), (300, 512, 16384)]:
        assert _plan("gemm", m, n, k).sum == "cluster" and _plan("gemm", m, n, k).kernel == "wide"
        assert lib.b200_w8a8_block_fp8_gemm_workspace_bytes(m, n, k) == 0, (m, n, k)
    for m in (1, 16, 33, 64, 100, 203, 256, 300, 700, 2000):
        for n, k in [(64, 8192), (200, 4096), (1024, 8192), (4096, 1792), (2112, 7168), (4096, 14336), (28672, 4096)]:
            p = _plan("gemm", m, n, k)
            need = p.splits * m * n * 4 if p.sum == "memory" else 0
            assert lib.b200_w8a8_block_fp8_gemm_workspace_bytes(m, n, k) >= need, (m, n, k, p)


def test_linear_wants_a_workspace_only_for_two_launches():
    """Without one, a size that runs as quantiser and GEMM is refused before anything is launched."""
    from sglang_b200 import _native as N

    lib, fake = N.load(), 1 << 20  # never read
    for m, n, k in [(9, 4096, 4096), (8, 5120, 5120), (203, 4096, 4096), (1027, 4096, 4096)]:
        assert not _plan("linear", m, n, k).kernel.endswith("quant")
        assert lib.b200_w8a8_block_fp8_linear(fake, N.BF16, fake, fake, fake, m, n, k, None, 0, None) == N.E_WORKSPACE
