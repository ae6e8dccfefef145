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
        for entry in ("gemm", "fanout", "linear"):
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
