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
