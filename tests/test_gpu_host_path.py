"""What the native host path hands back to the Python functions instead of running it itself."""
import pytest
import torch
import torch.autograd.forward_ad as fw

from rgd_triton_b200 import ops
from tests._util import gen, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["x", "w"])
def test_forward_mode_is_refused_for_rows(which):
    """The operators have no jvp: a tangent on an input that wants a gradient is an error, not dropped."""
    m = ops.FusedRMSNorm(64).cuda()
    x = randn(gen(0), 2, 5, 64).cuda().requires_grad_(True)
    with fw.dual_level():
        t = x if which == "x" else m.weight
        dual = fw.make_dual(t, torch.ones_like(t))
        with pytest.raises(RuntimeError):
            if which == "x":
                m(dual)
            else:
                torch.func.functional_call(m, {"weight": dual}, (x,))


@pytest.mark.parametrize("op", ["headln", "attn"])
def test_forward_mode_is_refused_for_heads(op):
    q, k, v = (randn(gen(i), 2, 8, 3, 64, dtype=torch.float16).cuda().requires_grad_(True) for i in range(3))
    with fw.dual_level():
        dual = fw.make_dual(q, torch.ones_like(q))
        with pytest.raises(RuntimeError):
            ops.FusedHeadLayerNorm()(dual, k, False) if op == "headln" else ops.FlashAttention()(dual, k, v)
