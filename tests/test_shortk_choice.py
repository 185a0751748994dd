"""Which kernel the BF16 precisions take for a short K on a 2-D C: the CUDA
cores' short-K kernel up to K = 28 in plans of their own; past that, and in
groups (whose CUDA-core lane has no short-K kernel), what the time model says."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.grouped import Group
from tccg_b200.plan import Plan

pytestmark = pytest.mark.gpu


def _con(k, m=4949, n=2080):
    return make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k))


@pytest.mark.parametrize("precision", ["bf16", "bf16x3"])
def test_choice(cuda, precision):
    assert "simt_shortk" in Plan(_con(28), precision).describe()
    assert "gett_tc" in Plan(_con(29), precision).describe()
    grp = Group([_con(24), _con(32)], precision)
    for p in grp.plans:
        assert "gett_tc" in p.describe()
