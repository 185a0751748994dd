"""FP32 calls whose C goes out in short runs (its stride-one M mode is short and
directly followed by the first N mode) take the tensor cores only where K makes
up for their slower epilogue."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,kernel", [(256, "simt_gett"), (1536, "gett_tc<F32X6>")])
def test_runs(cuda, k, kernel):
    runs = make_contraction("lykx", "kilj", "ixyj", dict(l=8, k=128, y=64, x=32, i=16, j=k // 16))
    assert kernel in Plan(runs, "fp32").describe()


def test_dense(cuda):
    assert "gett_tc<F32X6>" in Plan(make_contraction("mn", "mk", "kn", dict(m=1024, n=2048, k=256)), "fp32").describe()
