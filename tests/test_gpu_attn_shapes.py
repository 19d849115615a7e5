"""Attention at the edges of the kernels' dispatch: head dims that are multiples of 8, vector biases of
every alignment, causal grids of more heads than one scheduling group, few queries."""
import pytest
import torch

from rgd_triton_b200 import _lib, functional as F_
from tests._util import DTYPES, attention_backward, gen, randn
from tests.test_gpu_attn import check, make_bias

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_expired_waits():
    yield
    assert _lib.load().rgd_device_status() == 0


def _inputs(g, B, tq, tk, H, d, dtype):
    return (randn(g, B, tq, H, d, dtype=dtype), randn(g, B, tk, H, d, dtype=dtype), randn(g, B, tk, H, d, dtype=dtype),
            randn(g, B, tq, H, d, dtype=dtype))


@pytest.mark.parametrize("mode", ["single_pass", "two_kernel"])
@pytest.mark.parametrize("d", [8, 24, 56, 72, 104, 120])
@pytest.mark.parametrize("kind", [None, "vector", "matrix"])
def test_head_dims_that_are_multiples_of_8(d, kind, mode):
    """Channels past d are zero-filled tiles on the tensor-memory kernels: nothing of them may reach the
    outputs, and nothing past d channels may be written (the row after the last head is checked by the
    dense layout: an overrun would land in the next head's outputs)."""
    g = gen(d)
    for tq, tk in [(130, 136), (257, 96)]:
        q, k, v, do = _inputs(g, 2, tq, tk, 3, d, torch.bfloat16)
        bias = None if kind is None else make_bias(g, kind, 2, 3, tq, tk, torch.bfloat16)
        with attention_backward(mode):
            check(q, k, v, do, bias, False, f"d={d} {kind} ({tq},{tk})")


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("tk", [127, 128, 129, 260, 390])
def test_vector_bias_of_any_alignment(dt, d, tk):
    """Key counts around the 128-key block; a vector whose batch rows are not 16-byte addressable is staged
    by the compute threads, an aligned one by bulk copies."""
    g = gen(tk + d)
    q, k, v, do = _inputs(g, 2, 140, tk, 2, d, DTYPES[dt])
    bias = make_bias(g, "vector", 2, 2, 140, tk, DTYPES[dt])
    with attention_backward("two_kernel"):
        check(q, k, v, do, bias, False, f"vector d={d} tk={tk}")


@pytest.mark.parametrize("d,H", [(128, 100), (64, 200)])
def test_causal_grid_of_more_heads_than_a_group(d, H):
    """The causal grids interleave the query blocks of as many heads as fit L2; with more heads than that
    every head must still get exactly its own blocks: bit-equal to evaluating the heads in two halves."""
    g = gen(H)
    q, k, v, do = (t.cuda() for t in _inputs(g, 1, 300, 1030, H, d, torch.bfloat16))

    def run(sl):
        a, b, c = (t[:, :, sl].contiguous().requires_grad_(True) for t in (q, k, v))
        o = F_.flash_attn_func(a, b, c, None, True)
        return (o.detach(), *torch.autograd.grad(o, (a, b, c), do[:, :, sl].contiguous()))
    with attention_backward("two_kernel"):
        whole = run(slice(0, H))
        halves = [run(slice(0, H // 2)), run(slice(H // 2, H))]
    for w, x, y in zip(whole, *halves):
        assert torch.equal(w, torch.cat([x, y], dim=2))


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("d", [8, 40, 64, 96, 128])
@pytest.mark.parametrize("kind", [None, "vector", "matrix", "matrix_f32"])
def test_few_queries(dt, d, kind):
    """At most 16 queries: the split-key kernel.  Query counts around its 8-row halves, key counts around its
    16-key tiles and from one tile (one CTA) to enough for every cluster size."""
    dtype = DTYPES[dt]
    g = gen(d)
    for tq, tk in [(1, 1), (1, 15), (2, 16), (8, 17), (9, 64), (16, 129), (3, 1000), (16, 2100)]:
        q, k, v, do = _inputs(g, 2, tq, tk, 3, d, dtype)
        bias = None if kind is None else make_bias(g, kind, 2, 3, tq, tk, dtype)
        check(q, k, v, do, bias, False, f"few d={d} {kind} ({tq},{tk})")


def test_few_queries_many_heads_and_masked_keys():
    """More heads than CTAs the chip holds (other split), K / V expanded over the batch (stride 0), a fully
    masked first half of the keys (a warp whose tiles are all masked contributes nothing)."""
    g = gen(5)
    B, H, tk, d = 5, 70, 300, 64
    q = randn(g, B, 4, H, d, dtype=torch.float16).cuda()
    k, v = (randn(g, 1, tk, H, d, dtype=torch.float16).cuda().expand(B, tk, H, d) for _ in range(2))
    bias = torch.zeros(B, 1, 1, tk, dtype=torch.float16)
    bias[..., :150] = float("-inf")
    got = F_.flash_attn_func(q, k, v, bias.cuda())
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float()) / d ** 0.5 + bias.cuda().float()
    want = torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1), v.float())
    # P and the output are rounded to fp16: two half-ulp roundings of values of magnitude < 4
    assert (got.float() - want).abs().max().item() < 4 * 2 ** -10


@pytest.mark.parametrize("d", [40, 64, 96, 128])
@pytest.mark.parametrize("tq,tk", [(5, 40), (130, 200)])
@pytest.mark.parametrize("kind", ["vector", "matrix", "matrix_f32"])
def test_rows_masked_with_the_lowest_value(d, tq, tk, kind):
    """One sequence masked by the type's lowest value in every key (its product with log2(e) overflows fp32):
    its output is the mean of V, its gradients finite; the other sequence is as without a mask."""
    g = gen(d + tq)
    q, k, v, do = (t.cuda() for t in _inputs(g, 2, tq, tk, 3, d, torch.bfloat16))
    dt = torch.float32 if kind == "matrix_f32" else torch.bfloat16
    bias = torch.zeros(2, 1, 1 if kind == "vector" else tq, tk, dtype=dt, device="cuda")
    bias[1] = torch.finfo(dt).min

    def run(b):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        o = F_.flash_attn_func(*leaves, b)
        return [o.detach(), *torch.autograd.grad(o, leaves, do)]
    got, plain = run(bias), run(None)
    want = v[1].float().mean(0, keepdim=True).expand(tq, -1, -1)
    # P (1 here) is exact, the output is rounded to bf16: half an ulp of values below 2
    assert (got[0][1].float() - want).abs().max().item() < 2.0 ** -8
    for a, b in zip(got, plain):
        assert torch.isfinite(a).all()
        # two kernels' roundings of P and dS to bf16, summed over up to 200 keys or queries
        assert (a[0].float() - b[0].float()).norm() <= 1e-2 * b[0].float().norm()


@pytest.mark.parametrize("tq,d", [(3, 8), (3, 64), (3, 96), (3, 128), (130, 8), (130, 40), (130, 96)])
def test_largest_probability_is_not_rounded(tq, d):
    """A row whose maximum grows by 7.44 (log2) from one key block to a later one of the same warp: against a
    reference that lags behind, the largest probability would be 173.5 and rounded to 8 bits (0.29 % off)."""
    g = gen(d)
    H = 16
    q, k = torch.zeros(1, tq, H, d), torch.zeros(1, 640, H, d)
    q[..., 0], k[..., 0], k[:, 0, :, 0], k[:, 512, :, 0] = 1.0, -40.0, -5.15625, 0.0
    v = randn(g, 1, 640, H, d, dtype=torch.bfloat16)
    got = F_.flash_attn_func(q.bfloat16().cuda(), k.bfloat16().cuda(), v.cuda(), softmax_scale=1.0).cpu().double()
    p = k[0, :, 0, 0].double().softmax(0)
    want = torch.einsum("k,bkhd->bhd", p, v.double())[:, None].expand_as(got)
    # What is left is the rounding of the output: within half an ulp, evenly spread, 2^-8 / sqrt(3) at the foot of a
    # binade and half of it at its top, 0.41 * 2^-8 in the mean square.  The lagging reference gave 0.97 * 2^-8.
    assert ((got - want) / want).pow(2).mean().sqrt() <= 0.55 * 2.0 ** -8


def _masked_rows_reference(q, k, v, do, bias, causal, far):
    """Output and gradients in 64 bits, with the probabilities of the rows in `far` even over their largest bias."""
    q, k, v, do, bias = (t.double() for t in (q, k, v, do, bias))
    scale = q.shape[-1] ** -0.5
    bias = bias.expand(q.shape[0], q.shape[2], q.shape[1], k.shape[1])
    if causal:
        bias = bias.masked_fill(torch.ones(bias.shape[2:], dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    p = (torch.einsum("bqhd,bkhd->bhqk", q, k) * scale + bias).softmax(-1)
    even = (bias == bias.amax(-1, keepdim=True)).double()
    p = torch.where(far, even / even.sum(-1, keepdim=True), p)
    o = torch.einsum("bhqk,bkhd->bqhd", p, v)
    ds = p * (torch.einsum("bqhd,bkhd->bhqk", do, v) - torch.einsum("bqhd,bqhd->bhq", o, do)[..., None])
    return (o, scale * torch.einsum("bhqk,bkhd->bqhd", ds, k), scale * torch.einsum("bhqk,bqhd->bkhd", ds, q),
            torch.einsum("bhqk,bqhd->bkhd", p, do), ds)


@pytest.mark.parametrize("mode", ["single_pass", "two_kernel"])
@pytest.mark.parametrize("d", [20, 40, 64, 96, 128])
@pytest.mark.parametrize("tq,tk,causal", [(5, 40, False), (130, 200, False), (200, 1, False), (70, 65, False), (130, 130, True)])
@pytest.mark.parametrize("kind", ["vector", "matrix", "matrix_f32"])
@pytest.mark.parametrize("mask", [-1e9, "lowest"])
def test_gradients_of_rows_masked_far_down(mode, d, tq, tk, causal, kind, mask):
    """Rows whose every key carries a mask so large that one fp32 log-sum-exp no longer resolves the probabilities:
    all rows of a sequence, some rows of another (matrix bias), and rows in which one key carries it and the others
    -inf.  Output and gradients are those of even probabilities over the largest bias, on every kernel."""
    g = gen(d + tq)
    B, H = 3, 2
    q, k, v, do = (t.cuda() for t in _inputs(g, B, tq, tk, H, d, torch.bfloat16))
    dt = torch.float32 if kind == "matrix_f32" else torch.bfloat16
    low = torch.finfo(dt).min if mask == "lowest" else mask
    bias = randn(g, B, 1, 1 if kind == "vector" else tq, tk, dtype=dt).cuda()
    far = torch.zeros(B, 1, tq, 1, dtype=torch.bool, device="cuda")
    bias[1], far[1] = low, True
    if kind != "vector":
        bias[0, :, 1:4], far[0, :, 1:4] = low, True
    bias[2], far[2] = float("-inf"), True
    bias[2, ..., 0 if causal else tk // 2] = low
    want = _masked_rows_reference(q, k, v, do, bias, causal, far)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    with attention_backward(mode):
        o = F_.flash_attn_func(*leaves, bias, causal)
        got = [o.detach(), *torch.autograd.grad(o, leaves, do)]
    with_dbias = leaves + [bias.clone().requires_grad_(True)]
    with attention_backward(mode):
        o = F_.flash_attn_func(*with_dbias, causal)
        grads = torch.autograd.grad(o, with_dbias, do)
    for a, b in zip(got[1:], grads):
        assert (a - b).float().norm() <= 1e-2 * b.float().norm() + 1e-4 * b.numel() ** 0.5
    got.append(grads[3])
    ds = want[4].sum(1, keepdim=True)
    want = [*want[:4], ds.sum(2, keepdim=True) if kind == "vector" else ds]
    for name, a, b in zip(("o", "dq", "dk", "dv", "dbias"), got, want):
        for i in range(B):
            # P and dS are rounded to bf16 (2^-9 in the mean square), the results once more; what cancels to nothing
            # (dS of a row with one key) is left at the rounding of o in delta, 2^-9 of |dO| |o| per row
            err, ref = (a[i].double() - b[i]).norm().item(), b[i].norm().item()
            assert err <= 1e-2 * ref + 2e-3 * b[i].numel() ** 0.5 * (name != "o" and name != "dv"), (name, i, err, ref)


@pytest.mark.parametrize("d", [8, 40, 56])
@pytest.mark.parametrize("kind", [None, "vector"])
def test_small_problems_of_small_head_dims_are_reproducible(d, kind):
    """Below 2^24 scores dQ of a head_dim under 64 does not depend on the order of additions: 16 key blocks that
    would each add to it give the same bits every time."""
    g = gen(d)
    q, k, v, do = (t.cuda() for t in _inputs(g, 2, 300, 2000, 12, d, torch.bfloat16))
    bias = None if kind is None else make_bias(g, kind, 2, 12, 300, 2000, torch.bfloat16).cuda()

    def run():
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        return torch.autograd.grad(F_.flash_attn_func(*leaves, bias), leaves, do)
    first = run()
    for _ in range(5):
        for a, b in zip(run(), first):
            assert torch.equal(a, b)


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("what", ["expanded", "odd_offset", "summed"])
def test_large_problems_of_other_head_dims_copy_what_is_not_addressable(what, native, monkeypatch):
    """Keys and values expanded over the heads, a slice at an odd offset, an upstream gradient of stride 0: the same
    kernels run as on dense tensors, shown by the same bits."""
    if not native:
        monkeypatch.setattr(F_, "_bind_host", lambda t: None)
        monkeypatch.setattr(F_, "_HOST", None)
    g = gen(96)
    B, T, H, d = 2, 840, 12, 96
    q, k, v = (randn(g, B, T, H, d, dtype=torch.bfloat16).cuda() for _ in range(3))
    do = randn(g, B, T, H, d, dtype=torch.bfloat16).cuda()
    if what == "expanded":
        k, v = (t[:, :, :1].expand(B, T, H, d) for t in (k, v))
    elif what == "odd_offset":
        q = torch.cat([q.flatten(), q.flatten()[:8]])[1:-7].view(B, T, H, d)
    else:
        do = do[:, :1].expand(B, T, H, d)

    def run(dense):
        leaves = [(t.clone(memory_format=torch.contiguous_format) if dense else t.detach()).requires_grad_(True)
                  for t in (q, k, v)]
        with attention_backward("two_kernel"):
            o = F_.flash_attn_func(*leaves)
            return [o.detach(), *torch.autograd.grad(o, leaves, do.contiguous() if dense else do)]
    for a, b in zip(run(False), run(True)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("tq", [5, 130])
@pytest.mark.parametrize("kind", ["vector", "matrix", "matrix_odd"])
@pytest.mark.parametrize("dt,bias_dt", [("f16", "f16"), ("bf16", "bf16"), ("f16", "f32"), ("bf16", "f32")])
def test_bias_conversion_is_as_exact_as_one_rounding(tq, kind, dt, bias_dt):
    """One visible key and no score: the log-sum-exp is the key's bias, taken to base 2 and back."""
    g = gen(tq)
    B, H, tk = 8, 50, 9 if kind == "matrix_odd" else 8
    q, k, v, _ = (t.cuda() for t in _inputs(g, B, tq, tk, H, 64, DTYPES[dt]))
    value = (randn(g, B, H, 1 if kind == "vector" else tq) * 100).to(DTYPES[bias_dt])
    value[value == 0] = 1
    bias = torch.full((*value.shape, tk), float("-inf"), dtype=value.dtype)
    bias[..., 3] = value
    _, lse = F_.flash_attn_func(torch.zeros_like(q), k, v, bias.cuda(), return_lse=True)
    value = value.double().expand(B, H, tq)
    # the product is within 7.3e-8 (constant and rounding) of the exact one, the constant of the way back 0.3e-8 off,
    # its product rounded to 6.0e-8
    assert ((lse[:, :, :tq].cpu().double() - value) / value).abs().max() <= 1.37e-7


def test_a_bias_is_not_scanned_on_its_first_call():
    """Also where the call passes through the dispatch twice (keys and values that are copied first)."""
    from rgd_triton_b200 import ops
    g = gen(1)
    q = randn(g, 2, 1024, 8, 96, dtype=torch.float16).cuda()
    k, v = (randn(g, 2, 1024, 1, 96, dtype=torch.float16).cuda().expand(2, 1024, 8, 96) for _ in range(2))
    bias = torch.full((1, 1, 1024, 1024), -1e4, dtype=torch.float16).triu(1).cuda()
    m = ops.FlashAttention()
    for sight in range(3):
        m(q, k, v, bias)
        assert torch.is_tensor(m.cache._tiles[2]) == (sight > 0)


@pytest.mark.parametrize("d,H", [(128, 101), (64, 201)])
def test_causal_grid_of_more_heads_than_a_group_of_long_queries(d, H):
    """As above for the dK/dV kernel, whose groups are sized by Q and dO: 95 / 190 heads of 1030 queries fit one.  Two
    groups, one head apart in size."""
    g = gen(H + 1)
    q, k, v, do = (t.cuda() for t in _inputs(g, 1, 1030, 300, H, d, torch.bfloat16))

    def run(sl):
        a, b, c = (t[:, :, sl].contiguous().requires_grad_(True) for t in (q, k, v))
        o = F_.flash_attn_func(a, b, c, None, True)
        return (o.detach(), *torch.autograd.grad(o, (a, b, c), do[:, :, sl].contiguous()))
    with attention_backward("two_kernel"):
        whole = run(slice(0, H))
        halves = [run(slice(0, H // 2)), run(slice(H // 2, H))]
    for w, x, y in zip(whole, *halves):
        assert torch.equal(w, torch.cat([x, y], dim=2))


@pytest.mark.parametrize("d,single", [(d, False) for d in (8, 24, 56, 72, 104, 120)] + [(d, True) for d in (8, 24, 56)])
@pytest.mark.parametrize("kind", [None, "vector", "matrix"])
def test_nothing_is_written_past_the_channels(d, single, kind):
    """Outputs whose rows lie 8 elements further apart than they are long: the gaps and both ends stay as they
    were, forward (few and many queries) and backward."""
    import ctypes as C
    lib, bf = _lib.load(), torch.bfloat16
    g = gen(d)
    # with 2^24 scores and more the single-pass form exists for these head dims
    for B, H, tq, tk in ([(1, 2, 2900, 2896)] if single else [(2, 3, 5, 40), (2, 3, 130, 136)]):
        q, k, v, do = (t.cuda() for t in _inputs(g, B, tq, tk, H, d, bf))
        bias = None if kind is None else make_bias(g, kind, B, H, tq, tk, bf).cuda()
        bias_s = F_._prep_bias(bias, q, tq, tk)[1]
        lse = torch.empty(B, H, lib.rgd_attn_lse_rows(tq), device="cuda")
        bufs = [torch.full((B * n * H * (d + 8) + 16,), 7.0, dtype=bf, device="cuda") for n in (tq, tq, tk, tk)]
        outs = [b[8:-8].view(B, n, H, d + 8)[..., :d] for b, n in zip(bufs, (tq, tq, tk, tk))]
        ref = lambda t: C.byref(F_._attn_heads(t))
        o, dq, dk, dv = outs
        stream = torch.cuda.current_stream().cuda_stream
        assert lib.rgd_attn_fwd(ref(q), ref(k), ref(v), C.byref(bias_s), ref(o), lse.data_ptr(), B, H, tq, tk, d, d ** -0.5, 0,
                                _lib.RGD_BF16, None, stream) == 0
        size = lib.rgd_attn_bwd_single_pass_workspace_bytes if single else lib.rgd_attn_bwd_workspace_bytes
        work = torch.empty(size(B, H, tq, tk, d, _lib.RGD_BF16), dtype=torch.uint8, device="cuda")
        assert lib.rgd_attn_bwd(ref(q), ref(k), ref(v), C.byref(bias_s), ref(o), lse.data_ptr(), ref(do), ref(dq), ref(dk),
                                ref(dv), B, H, tq, tk, d, d ** -0.5, 0, _lib.RGD_BF16, work.data_ptr(), work.numel(), None,
                                stream) == 0
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        with attention_backward("single_pass" if single else "two_kernel"):
            want = F_.flash_attn_func(*leaves, bias)
            grads = torch.autograd.grad(want, leaves, do)
        for i, (a, b) in enumerate(zip(outs, (want, *grads))):
            # dQ of the single-pass form is summed in no fixed order: one rounding step of the largest value
            assert torch.equal(a, b) or (single and i == 1 and (a - b).abs().max() <= 2.0 ** -8 * b.abs().max())
        for b, n in zip(bufs, (tq, tq, tk, tk)):
            assert (b[:8] == 7).all() and (b[-8:] == 7).all() and (b[8:-8].view(B, n, H, d + 8)[..., d:] == 7).all()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("tk", [1, 40, 60, 65, 190, 193])
def test_fp32_bias_with_half_a_block_past_the_keys(d, tk):
    """A matrix bias that the threads read themselves: a block whose second 64 keys lie past the end reads nothing there
    (the bias ends with its allocation's last row)."""
    g = gen(tk)
    q, k, v, do = _inputs(g, 2, 130, tk, 3, d, torch.bfloat16)
    check(q, k, v, do, make_bias(g, "matrix_f32", 2, 3, 130, tk, torch.bfloat16), False, f"d={d} tk={tk}")


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("H", [37, 75])
def test_few_queries_around_the_heads_that_fill_the_chip(d, H):
    """148 and 150 heads x sequences: the last that are split over a cluster by the room left, the first that are not."""
    g = gen(H)
    for tq, tk in [(1, 640), (16, 1030)]:
        q, k, v, do = _inputs(g, 4 if H == 37 else 2, tq, tk, H, d, torch.bfloat16)
        check(q, k, v, do, None, False, f"few H={H} d={d} ({tq},{tk})")


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("d", [96, 100])
def test_large_outputs_of_other_head_dims_are_dense(d, native, monkeypatch):
    """Whatever the layout of q (heads second here): its heads and channels can be viewed as one dimension."""
    if not native:
        monkeypatch.setattr(F_, "_bind_host", lambda t: None)
        monkeypatch.setattr(F_, "_HOST", None)
    g = gen(d)
    B, T, H = 2, 840, 12
    heads_second = [randn(g, B, H, T, d, dtype=torch.bfloat16).cuda() for _ in range(3)]
    q, k, v = (t.transpose(1, 2).requires_grad_(True) for t in heads_second)
    o = F_.flash_attn_func(q, k, v)
    assert o.view(B, T, H * d).shape == (B, T, H * d)
    grads = torch.autograd.grad(o, (q, k, v), torch.ones_like(o))
    assert [t.shape for t in grads] == [q.shape] * 3
    if native:
        assert all(t.is_contiguous() for t in grads)
    dense = F_.flash_attn_func(*(t.transpose(1, 2).contiguous() for t in heads_second))
    assert torch.equal(o, dense)
