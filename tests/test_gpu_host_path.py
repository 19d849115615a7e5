"""What the native host path hands back to the Python functions instead of running it itself."""
import pytest
import torch
import torch.autograd.forward_ad as fw

from rgd_triton_b200 import functional as F_, ops
from tests._util import attention_backward, gen, randn, rotary_table

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


# ---------------------------------------------------------------------------------------------- autograd around the calls
def _calls():
    """name -> (call, inputs that want a gradient): every operator on ordinary shapes of the native path."""
    g = gen(3)
    f16 = torch.float16
    x, y = randn(g, 2, 9, 64).cuda(), randn(g, 2, 5, 96).cuda()
    q, k = randn(g, 2, 40, 3, 64, dtype=f16).cuda(), randn(g, 2, 24, 3, 64, dtype=f16).cuda()
    v = randn(g, 2, 24, 3, 64, dtype=f16).cuda()
    bias = randn(g, 2, 3, 40, 24, dtype=f16).cuda()
    pos = rotary_table(64, 32, f16).cuda()
    rms, rms2 = ops.FusedRMSNorm(64).cuda(), ops.FusedRMSNorm2((64, 96)).cuda()
    l2, l22, ln, rope, lnrope, attn = (ops.L2Normalize(), ops.FusedL2Normalize2(), ops.FusedHeadLayerNorm(), ops.RoPE(),
                                       ops.FusedLNRoPE(), ops.FlashAttention())
    return {"l2": (lambda a: l2(a), [x]), "l2x2": (lambda a, b: l22(a, b), [x, y]),
            "rms": (rms, [x]), "rms2": (lambda a, b: rms2(a, b), [x, y]),
            "headln": (lambda a, b: ln(a, b, False), [q, k]), "rope": (lambda a, b: rope(a, b, pos, 20, False), [q, k]),
            "lnrope": (lambda a, b: lnrope(a, b, pos, (20, 24), False), [q, k]),
            "attn": (lambda a, b, c: attn(a, b, c), [q, k, v]), "attn_bias": (lambda a, b, c: attn(a, b, c, bias), [q, k, v])}


CALLS = ["l2", "l2x2", "rms", "rms2", "headln", "rope", "lnrope", "attn", "attn_bias"]


def _grads(call, inputs, wrap=lambda f: f):
    leaves = [t.clone().requires_grad_(True) for t in inputs]
    with attention_backward("two_kernel"):      # bit-reproducible, so that two ways can be compared exactly
        out = wrap(call)(*leaves)
        outs = out if isinstance(out, tuple) else (out,)
        grads = torch.autograd.grad(outs, leaves, [torch.cos(o.detach().float()).to(o.dtype) for o in outs])
    return [o.detach() for o in outs] + list(grads)


@pytest.mark.parametrize("name", CALLS)
def test_checkpoint(name):
    """torch.utils.checkpoint stops its recomputation by an exception out of the pack hook of the region's last
    saved tensor, which here is one of the operator's own."""
    from torch.utils.checkpoint import checkpoint
    call, inputs = _calls()[name]
    want = _grads(call, inputs)
    got = _grads(call, inputs, lambda f: lambda *a: checkpoint(f, *a, use_reentrant=False))
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", CALLS)
def test_pack_hooks_raise_their_own_exception(name):
    call, inputs = _calls()[name]

    def pack(t):
        raise KeyError("packed")
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        with pytest.raises(KeyError, match="packed"):
            call(*[t.clone().requires_grad_(True) for t in inputs])


def _dense_copies(call, inputs):
    """_grads with every saved tensor replaced by a dense copy of itself, as save_on_cpu does."""
    with torch.autograd.graph.save_on_cpu():
        return _grads(call, inputs)


@pytest.mark.parametrize("name", ["rms", "rope", "lnrope", "attn_slice", "attn_transposed", "attn_q"])
def test_saved_tensors_that_come_back_dense(name):
    """Strided weights, rotary tables, biases and queries: the backward has to read the copies it unpacks by their
    own strides."""
    g = gen(6)
    f16 = torch.float16
    calls = _calls()
    if name == "rms":
        w = (1 + 0.1 * randn(g, 2, 3, 64)).cuda()[:, 1:2]           # [B, 1, C] of a [B, 3, C] modulation
        m = ops.FusedRMSNorm(64, elementwise_affine=False)
        call, inputs = lambda a, w: m(a, w), [calls["rms"][1][0], w]
        base = _grads(call, [inputs[0], w.contiguous()])
        got = _dense_copies(lambda a, big: m(a, big[:, 1:2]), [inputs[0], w.expand(2, 3, 64).contiguous()])
        got[2] = got[2][:, 1:2]
    elif name in ("rope", "lnrope"):
        table = rotary_table(80, 48, f16).cuda()[:, 5:70, :32]
        m = ops.RoPE() if name == "rope" else ops.FusedLNRoPE()
        call, inputs = lambda a, b: m(a, b, table, 20, False), calls[name][1]
        base, got = _grads(call, inputs), _dense_copies(call, inputs)
    else:
        m = ops.FlashAttention()
        inputs = calls["attn"][1]
        bias = {"attn_slice": randn(g, 2, 3, 64, 64, dtype=f16).cuda()[:, :, 8:48, 16:40],
                "attn_transposed": randn(g, 3, 2, 40, 24, dtype=f16).cuda().transpose(0, 1), "attn_q": None}[name]
        if name == "attn_q":
            call = lambda a, b, c: m(a.transpose(1, 2).contiguous().transpose(1, 2), b, c)
        else:
            call = lambda a, b, c: m(a, b, c, bias)
        base, got = _grads(call, inputs), _dense_copies(call, inputs)
    for a, b in zip(got, base):
        assert torch.equal(a, b)


@pytest.mark.parametrize("native", [True, False])
def test_tile_lists_of_a_bias_that_comes_back_dense(native, monkeypatch):
    """An expanded bias has one slice of tile lists; its dense copy would index one per (batch, head)."""
    if not native:
        monkeypatch.setattr(F_, "_bind_host", lambda t: None)
        monkeypatch.setattr(F_, "_HOST", None)
    g = gen(7)
    f16 = torch.float16
    q, k, v = (randn(g, 2, 1024, 2, 64, dtype=f16).cuda() for _ in range(3))
    bias = torch.zeros(1024, 1024, dtype=f16)
    bias[:512, 512:] = -1e4
    bias = bias.cuda().expand(2, 2, 1024, 1024)
    m = ops.FlashAttention()
    call = lambda a, b, c: m(a, b, c, bias)
    base = [_grads(call, [q, k, v]) for _ in range(3)][-1]
    assert torch.is_tensor(m.cache._tiles[2])
    for a, b in zip(_dense_copies(call, [q, k, v]), base):
        assert torch.equal(a, b)


def test_saved_tensors_of_another_shape_are_refused():
    call, inputs = _calls()["attn_bias"]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t[..., :8] if t.dim() == 4 else t):
        out = call(*[t.clone().requires_grad_(True) for t in inputs])
        with pytest.raises(RuntimeError, match="saved tensor"):
            out.sum().backward()


# ---------------------------------------------------------------------------------------------- callers that watch the operations
@pytest.mark.parametrize("name", CALLS)
def test_compiled_autograd(name):
    """Forward eagerly, backward traced by compiled autograd, also after a change of sizes and of a constant."""
    from torch._dynamo import compiled_autograd

    def grads(call, inputs, compiled):
        leaves = [t.clone().requires_grad_(True) for t in inputs]
        with attention_backward("two_kernel"):
            out = call(*leaves)
            outs = out if isinstance(out, tuple) else (out,)
            gs = [torch.cos(o.detach().float()).to(o.dtype) for o in outs]
            if compiled:
                with compiled_autograd._enable(lambda gm: torch.compile(gm, backend="eager")):
                    torch.autograd.backward(outs, gs)
            else:
                torch.autograd.backward(outs, gs)
        return [t.grad for t in leaves]
    call, inputs = _calls()[name]
    smaller = inputs if name == "attn_bias" else [t[:, :5] for t in inputs]
    pos = rotary_table(64, 32, torch.float16).cuda()
    other = (lambda a, b: ops.RoPE()(a, b, pos, 3, False)) if name == "rope" else call
    torch._dynamo.reset()
    for f, ins in [(call, inputs), (call, smaller), (other, inputs)]:
        for a, b in zip(grads(f, ins, True), grads(f, ins, False)):
            assert torch.equal(a, b)


@pytest.mark.filterwarnings("ignore")       # of the tracer: sizes that become constants, its own deprecation
@pytest.mark.parametrize("name", ["l2", "rms", "headln", "rope", "attn"])
def test_jit_trace(name):
    call, inputs = _calls()[name]
    leaves = [t.clone().requires_grad_(True) for t in inputs]
    traced = torch.jit.trace(call, tuple(leaves), check_trace=False)
    fresh = [t.flip(1).clone() for t in inputs]
    for a, b in zip(_grads(traced, fresh), _grads(call, fresh)):
        assert torch.equal(a, b)


def test_dispatch_modes_and_transforms():
    """A dispatch mode sees the operator's allocations; a transform, which the operators have no rule for, is refused."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.ops = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.ops.append(func)
            return func(*args, **(kwargs or {}))
    call, (x,) = _calls()["l2"]
    with Seen() as seen:
        y = call(x)
    assert seen.ops and torch.equal(y, call(x))
    with pytest.raises(RuntimeError):
        torch.func.vmap(call)(x[None])
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: call(t).sum())(x)


@pytest.mark.parametrize("arg", ["causal", "heads_second"])
def test_flags_without_a_truth_value(arg):
    """What bool() of the argument raises is what the call raises."""
    q, k, v = _calls()["attn"][1]
    with pytest.raises(RuntimeError, match="[Bb]oolean value"):
        if arg == "causal":
            ops.FlashAttention()(q, k, v, None, torch.tensor([True, False]))
        else:
            ops.FusedHeadLayerNorm()(q, q, torch.tensor([True, False]))


# ---------------------------------------------------------------------------------------------- the native path against the Python one
ROUTES = ["native", "no_cache", "python"]


def _by_route(route, monkeypatch):
    """The same operators through the native path, without launch caches, or through the Python functions."""
    calls = _calls()
    if route == "no_cache":
        for call, _ in calls.values():
            for m in [call] + [c.cell_contents for c in (getattr(call, "__closure__", None) or ())]:
                if isinstance(m, ops.CachableModule):
                    m.enable_cache(False)
    if route == "python":
        monkeypatch.setattr(F_, "_bind_host", lambda t: None)
        monkeypatch.setattr(F_, "_HOST", None)
    return calls


@pytest.mark.parametrize("route", ROUTES[1:])
@pytest.mark.parametrize("name", CALLS)
def test_routes_agree(name, route, monkeypatch):
    """Checks, marshalling and workspaces exist twice, in C++ and in Python: same bits, dense and strided."""
    call, inputs = _calls()[name]
    strided = [torch.cat([t, t], dim=-2)[..., : t.shape[-2], :] for t in inputs]
    want = [_grads(call, ins) for ins in (inputs, strided)]
    other = _by_route(route, monkeypatch)[name][0]
    for ins, w in zip((inputs, strided), want):
        for a, b in zip(_grads(other, ins), w):
            assert torch.equal(a, b)


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("name", CALLS)
def test_two_backwards(name, route, monkeypatch):
    """A kept graph gives the same gradients again; a released one, and inputs changed in between, are errors."""
    call, inputs = _by_route(route, monkeypatch)[name]
    leaves = [t.clone().requires_grad_(True) for t in inputs]
    with attention_backward("two_kernel"):
        out = call(*leaves)
        outs = out if isinstance(out, tuple) else (out,)
        gs = [torch.ones_like(o) for o in outs]
        first = torch.autograd.grad(outs, leaves, gs, retain_graph=True)
        second = torch.autograd.grad(outs, leaves, gs)
    for a, b in zip(first, second):
        assert torch.equal(a, b)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(outs, leaves, gs)
    if name != "rope":              # saves no input
        out = call(*leaves)
        outs = out if isinstance(out, tuple) else (out,)
        with torch.no_grad():
            leaves[0].mul_(2)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            torch.autograd.grad(outs, leaves, gs)


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("name", ["l2x2", "rms2", "headln", "rope", "lnrope"])
def test_one_of_two_outputs_without_a_gradient(name, route, monkeypatch):
    """The input whose output nobody used gets zeros, the other one its gradient."""
    call, inputs = _by_route(route, monkeypatch)[name]
    leaves = [t.clone().requires_grad_(True) for t in inputs]
    outs = call(*leaves)
    g = torch.cos(outs[1].detach().float()).to(outs[1].dtype)
    used = torch.autograd.grad(outs[1], leaves, g)
    outs = call(*leaves)
    both = torch.autograd.grad(outs, leaves, [torch.zeros_like(outs[0]), g])
    assert not used[0].any()
    for a, b in zip(used, both):
        assert torch.equal(a, b)


@pytest.mark.parametrize("route", ROUTES)
def test_side_stream_and_thread(route, monkeypatch):
    """Forward and backward on a stream of their own, from another thread, through one module used by both threads."""
    import threading
    calls = _by_route(route, monkeypatch)
    want = {n: _grads(*calls[n]) for n in ("rms", "lnrope", "attn_bias")}
    torch.cuda.synchronize()
    failures = []

    def work():
        try:
            stream = torch.cuda.Stream()
            for _ in range(5):
                for n, w in want.items():
                    with torch.cuda.stream(stream):
                        leaves = [t.clone().requires_grad_(True) for t in calls[n][1]]
                        out = calls[n][0](*leaves)
                        outs = out if isinstance(out, tuple) else (out,)
                        got = [*outs, *torch.autograd.grad(outs, leaves, [torch.cos(o.detach().float()).to(o.dtype) for o in outs])]
                    stream.synchronize()
                    assert all(torch.equal(a, b) for a, b in zip(got, w))
        except BaseException as e:      # noqa: BLE001  (reported by the main thread)
            failures.append(e)
    with attention_backward("two_kernel"):
        threads = [threading.Thread(target=work) for _ in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not failures
