"""The tcgen05 backward kernel (``sa_attn_bwd_packed``) where its tiles, lists and planes have edges: against
``torch.autograd`` through SDPA on the host in fp32, and against the generic backward over the same lists."""
import pytest
import torch
import torch.nn.functional as F

import sparseattention_b200 as sa
import workloads
from sparseattention_b200 import _native

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _mask(kind, B, H, Sq, Sk, seed):
    g = torch.Generator().manual_seed(seed)
    if kind == "full":
        return torch.ones((1, 1, Sq, Sk), dtype=torch.bool)
    if kind == "bands":                                        # empty query blocks and kv blocks, single elements
        m = torch.zeros((B, 1, Sq, Sk), dtype=torch.bool)
        m[0, 0, 5, 3] = m[0, 0, Sq - 1, Sk - 1] = True
        m[-1, 0, Sq // 2:, : Sk // 3] = True
        return m
    keep = torch.rand((B, H, (Sq + 31) // 32, (Sk + 31) // 32), generator=g) < 0.3
    m = keep.repeat_interleave(32, 2).repeat_interleave(32, 3)[:, :, :Sq, :Sk]
    return m & (torch.rand((B, H, Sq, Sk), generator=g) < 0.9) if kind == "ragged" else m.clone()


def _inputs(B, H, Sq, Sk, D, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    new = lambda S: torch.randn((B, H, S, D), generator=g).to(dtype)
    return new(Sq), new(Sk), new(Sk), new(Sq)


def _check(got, want, what):
    """Gradients of 16-bit inputs: the forward's bound, relative to the largest entry (P, dS and the result are
    rounded to the type: 2^-9 of the value each in bf16)."""
    scale = max(1.0, want.abs().max().item())
    diff = (got.float().cpu() - want).abs()
    assert torch.isfinite(got).all() and diff.max().item() <= 2e-2 * scale and diff.mean().item() <= 2e-3 * scale, \
        f"{what}: max {diff.max().item():.3e} mean {diff.mean().item():.3e} scale {scale:.2f}"


@pytest.mark.parametrize("kind,B,H,Sq,Sk,D,bk,dtype", [
    ("full", 1, 2, 128, 32, 64, 32, torch.float16),            # smallest: one kv tile, three quarters of it past the end
    ("full", 2, 1, 256, 128, 128, 128, torch.bfloat16),
    ("bands", 2, 2, 384, 352, 128, 32, torch.bfloat16),        # kv rows no multiple of 128, walks of 0 and 1 entries
    ("blocks", 1, 3, 640, 448, 64, 64, torch.float16),
    ("ragged", 2, 3, 256, 1184, 128, 32, torch.bfloat16),      # a mask per head
    ("ragged", 2, 1, 1152, 384, 64, 128, torch.bfloat16),
])
def test_gradients_at_the_edges_of_the_tiles(native_lib, kind, B, H, Sq, Sk, D, bk, dtype):
    q, k, v, w = _inputs(B, H, Sq, Sk, D, dtype, seed=Sq + Sk)
    mask = _mask(kind, B, H, Sq, Sk, seed=bk + D)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    out = F.scaled_dot_product_attention(qf, kf, vf, attn_mask=mask.expand(B, H, Sq, Sk))
    live = mask.any(-1, keepdim=True)
    torch.where(live, out, torch.zeros_like(out)).mul(w.float()).sum().backward()
    # projections as they come out of one fused matrix: [B, S, 3, H, D] views where the lengths agree
    leaves = [t.to(DEV).transpose(1, 2).contiguous().transpose(1, 2).requires_grad_(True) for t in (q, k, v)]
    sa.sparse_attention(*leaves, mask.to(DEV), 128, bk, check_status=True).backward(w.to(DEV))
    for name, leaf, ref in zip(("dq", "dk", "dv"), leaves, (qf.grad, kf.grad, vf.grad)):
        _check(leaf.grad, torch.nan_to_num(ref), f"{name} {kind} Sq={Sq} Sk={Sk} D={D} bk={bk}")


@pytest.mark.parametrize("Sq,Sk,D,dtype", [(4096, 256, 128, torch.bfloat16), (256, 4096, 64, torch.float16)])
def test_long_walks(native_lib, Sq, Sk, D, dtype):
    """32 steps that reuse the same columns of tensor memory for the scores, P, the other product and dS: any step that
    overwrote them early would show against the generic backward, or from one run to the next."""
    B, H = 3, 17                                               # 1734 tiles: every SM has several
    q, k, v, w = (t.to(DEV) for t in _inputs(B, H, Sq, Sk, D, dtype, seed=D))
    mask = _mask("ragged", B, 1, Sq, Sk, seed=D).to(DEV) | torch.rand((B, 1, Sq // 128, Sk // 128), device=DEV).lt(0.7) \
        .repeat_interleave(128, 2).repeat_interleave(128, 3)
    mask = mask.expand(B, H, Sq, Sk)
    md = sa.compute_mask_kernel(mask, 128, 32)
    lists = (md.unmasked_kv_ids, md.unmasked_lens, md.masked_kv_ids, md.masked_lens)
    o, lse = _native.attn_fwd_op(q, k, v, mask, md.packed_bits, *lists, 128, 32, _native.SA_IMPL_AUTO, False, True)
    want = _native._transposed_and_bwd(q, k, v, o, w, lse, None, mask, *lists, 128, 32)
    first = None
    for _ in range(4):
        got = _native.attn_grads_op(q, k, v, o, w, lse, None, mask, md.packed_bits, *lists, 128, 32)
        first = first or got
        for name, g, r, f in zip(("dq", "dk", "dv"), got, want, first):
            _check(g, r.float().cpu(), name)
            assert torch.equal(g, f), f"{name}: not the same twice"


@pytest.mark.parametrize("bk,per_head_lists", [(32, False), (64, True), (128, True)])
def test_caller_lists_that_differ_from_the_mask(native_lib, bk, per_head_lists):
    """Lists a caller has pruned and widened: the kernel follows the lists, as the generic backward does."""
    B, H, S, D = 2, 2, 512, 64
    q, k, v, w = (t.to(DEV) for t in _inputs(B, H, S, S, D, torch.bfloat16, seed=bk))
    mask = workloads.random_block_mask(B, S, 0.4, 0.3, seed=bk).to(DEV).expand(B, H, S, S)
    md = sa.compute_mask_kernel(mask, 128, bk)
    lists = [t.clone() if per_head_lists else t[:, :1].clone()
             for t in (md.unmasked_kv_ids, md.unmasked_lens, md.masked_kv_ids, md.masked_lens)]
    lists[1][0, 0, 1:] = torch.clamp(lists[1][0, 0, 1:] - 1, min=0)           # the last full block of some rows dropped
    lists[3][1, -1] = torch.clamp(lists[3][1, -1] - 1, min=0)                 # and the last partial one of others
    n = int(lists[1][1, 0, 2])                                                # a partial block declared full
    if int(lists[3][1, 0, 2]) > 0:
        lists[0][1, 0, 2, n] = lists[2][1, 0, 2, int(lists[3][1, 0, 2]) - 1]
        lists[1][1, 0, 2] += 1
        lists[3][1, 0, 2] -= 1
    lists = [t.expand(B, H, *t.shape[2:]) for t in lists]
    o, lse = _native.attn_fwd_op(q, k, v, mask, md.packed_bits, *lists, 128, bk, _native.SA_IMPL_AUTO, False, True)
    got = _native.attn_grads_op(q, k, v, o, w, lse, None, mask, md.packed_bits, *lists, 128, bk)
    want = _native._transposed_and_bwd(q, k, v, o, w, lse, None, mask, *lists, 128, bk)
    again = _native.attn_grads_op(q, k, v, o, w, lse, None, mask, md.packed_bits, *lists, 128, bk)
    for name, g, r, a in zip(("dq", "dk", "dv"), got, want, again):
        _check(g, r.float().cpu(), name)
        assert torch.equal(g, a), f"{name}: not the same twice"


def test_gradient_op_passes_opcheck(native_lib):
    B, H, S, D = 1, 2, 256, 64
    q, k, v, w = (t.to(DEV) for t in _inputs(B, H, S, S, D, torch.bfloat16, seed=5))
    mask = workloads.random_block_mask(B, S, 0.5, 0.2, seed=6).to(DEV)
    f_ids, f_lens, p_ids, p_lens, bits = _native.classify(mask, 128, 32)
    lists = [t.expand(B, H, *t.shape[2:]) for t in (f_ids, f_lens, p_ids, p_lens)]
    o, lse = _native.attn_fwd_op(q, k, v, mask.expand(B, H, S, S), bits, *lists, 128, 32, _native.SA_IMPL_AUTO, False, True)
    torch.library.opcheck(_native.attn_grads_op, (q, k, v, o, w, lse, torch.ones_like(lse), mask.expand(B, H, S, S), bits,
                                                  *lists, 128, 32), test_utils=("test_schema", "test_faketensor"))
    call, plan, ms = _native.plan_call(q, k, v, mask, 128, 32)
    o, lse, scratch = _native.run_call(q, k, mask, call, plan, ms, 32, True, False)
    torch.library.opcheck(_native.call_grads_op, (q, k, v, o, lse, scratch, w, None, list(ms), 128, 32, False),
                          test_utils=("test_schema", "test_faketensor"))


@pytest.mark.parametrize("caller_lists", [False, True])
def test_batched_and_watched_gradients(native_lib, caller_lists):
    """Several gradients at once (``is_grads_batched``, a vectorised Jacobian: vmap over the backward) equal them one by
    one, and a dispatch mode around the backward sees its op."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Watch(TorchDispatchMode):
        seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(func.namespace)
            return func(*args, **(kwargs or {}))

    B, H, S, D = 1, 2, 256, 64
    q, k, v, w = (t.to(DEV) for t in _inputs(B, H, S, S, D, torch.float16, seed=15))
    mask = workloads.random_block_mask(B, S, 0.5, 0.2, seed=16).to(DEV)
    leaves = [t.requires_grad_(True) for t in (q, k, v)]
    md = sa.compute_mask_kernel(mask.expand(B, H, S, S), 128, 32) if caller_lists else None
    out, lse = sa.sparse_attention(*leaves, mask, 128, 32, mask_metadata=md, return_lse=True)
    many = torch.stack([w, -w, w.flip(2)])
    many_lse = torch.randn((3, B, H, S), device=DEV)
    got = torch.autograd.grad((out, lse), leaves, (many, many_lse), is_grads_batched=True, retain_graph=True)
    for i in range(3):
        want = torch.autograd.grad((out, lse), leaves, (many[i], many_lse[i]), retain_graph=True)
        for name, g, r in zip(("dq", "dk", "dv"), got, want):
            assert torch.equal(g[i], r), name
    with Watch() as watch:
        watched = torch.autograd.grad((out, lse), leaves, (many[i], many_lse[i]))
    assert "sparseattention" in watch.seen and all(torch.equal(g, r) for g, r in zip(watched, want))
    row = lambda x: sa.sparse_attention(x, k, v, mask, 128, 32, mask_metadata=md)[0, 0, 7, :2].float()
    jac = torch.autograd.functional.jacobian(row, q.detach(), vectorize=True)
    assert torch.equal(jac, torch.autograd.functional.jacobian(row, q.detach())) and jac.abs().max().item() > 0


def test_differentiable_calls_in_the_forms_autograd_has(native_lib):
    """The one-call forward with gradients: from a fresh thread, with a gradient off a 16-byte boundary, under
    saved-tensor hooks, through the log-sum-exp alone, twice over one graph, and refused where it always was."""
    B, H, S, D = 1, 2, 256, 64
    q, k, v, w = (t.to(DEV) for t in _inputs(B, H, S, S, D, torch.float16, seed=9))
    mask = workloads.random_block_mask(B, S, 0.5, 0.2, seed=10).to(DEV)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    call = lambda **kw: sa.sparse_attention(*leaves, mask, 64, 32, **kw)
    out = call()
    want = torch.autograd.grad(out, leaves, w, retain_graph=True)
    shifted = torch.empty(w.numel() + 1, dtype=w.dtype, device=DEV)[1:].view(w.shape).copy_(w)
    results = [torch.autograd.grad(out, leaves, shifted, retain_graph=True), torch.autograd.grad(out, leaves, w)]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (t.cpu(), t.stride()), lambda p: p[0].to(DEV)):
        out = call()
    results.append(torch.autograd.grad(out, leaves, w))
    strided = [t.transpose(1, 2).contiguous().transpose(1, 2).detach().requires_grad_(True) for t in leaves]
    results.append(torch.autograd.grad(sa.sparse_attention(*strided, mask, 64, 32), strided, w))
    # the registered ops, over lists made before
    md = sa.compute_mask_kernel(mask.expand(B, H, S, S), 128, 32)
    results.append(torch.autograd.grad(sa.sparse_attention(*leaves, mask, 128, 32, mask_metadata=md), leaves, w))
    for got in results:
        for g, r in zip(got, want):
            assert torch.equal(g, r)
    lse = call(return_lse=True)[1]
    by_lse = torch.autograd.grad(lse, leaves[:2], torch.ones_like(lse))
    lse = sa.sparse_attention(*leaves, mask, 128, 32, mask_metadata=md, return_lse=True)[1]
    for g, r in zip(by_lse, torch.autograd.grad(lse, leaves[:2], torch.ones_like(lse))):
        assert torch.equal(g, r) and g.abs().max().item() > 0
    twice = torch.autograd.grad(call(), leaves, w, create_graph=True)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(twice[0].sum(), leaves[0])


@pytest.mark.parametrize("caller_lists", [False, True])
def test_a_backward_that_reports_raises(native_lib, caller_lists):
    """What the backward kernel reports in its status word reaches the caller that asked for it.  A kv-block id outside the
    tensor (the kernel checks each, and uses block 0) arrives in the saved lists through a saved-tensor hook."""
    B, H, S, D = 1, 2, 256, 64
    q, k, v, w = (t.to(DEV) for t in _inputs(B, H, S, S, D, torch.float16, seed=12))
    mask = torch.ones((B, H, S, S), dtype=torch.bool, device=DEV)
    leaves = [t.requires_grad_(True) for t in (q, k, v)]
    md = sa.compute_mask_kernel(mask, 128, 32) if caller_lists else None
    at = _native.plan_call(q.detach(), k.detach(), v.detach(), mask, 128, 32)[1][5] // 4        # where the full ids start

    def unpack(t):
        if caller_lists and t.dtype == torch.int32 and tuple(t.shape) == (B, H, S // 128, S // 32):
            t = t.clone()
            t[0, 0, 0, 0] = 1 << 20
        elif t.dtype == torch.uint8:
            t = t.clone()
            t.view(torch.int32)[at] = 1 << 20
        return t

    for check in (True, False):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            out = sa.sparse_attention(*leaves, mask, 128, 32, mask_metadata=md, check_status=check)
        if check:
            with pytest.raises(RuntimeError, match="out of range"):
                torch.autograd.grad(out, leaves, w)
        else:
            torch.autograd.grad(out, leaves, w)
    out = sa.sparse_attention(*leaves, mask, 128, 32, mask_metadata=md, check_status=True)
    assert all(torch.isfinite(g).all() for g in torch.autograd.grad(out, leaves, w))


@pytest.mark.parametrize("caller_lists", [False, True])
@pytest.mark.parametrize("what", ["lse", "out", "qkv", "lists"])
def test_saved_tensors_come_back_in_another_layout(native_lib, what, caller_lists):
    """A saved-tensor hook may hand back any tensor of equal values: transposed in memory, or every second element of a
    wider buffer.  Same gradients to the bit."""
    B, H, S, D = 1, 3, 384, 64
    q, k, v, w = (t.to(DEV) for t in _inputs(B, H, S, S, D, torch.bfloat16, seed=13))
    mask = _mask("ragged", B, 1, S, S, seed=14).to(DEV)
    leaves = [t.requires_grad_(True) for t in (q, k, v)]
    md = sa.compute_mask_kernel(mask.expand(B, H, S, S), 128, 32) if caller_lists else None
    is_input = lambda t: any(t.data_ptr() == x.data_ptr() for x in leaves)
    ours = {"lse": lambda t: t.dtype == torch.float32, "out": lambda t: t.dtype == torch.bfloat16 and not is_input(t),
            "qkv": is_input, "lists": lambda t: t.dtype in (torch.int32, torch.uint8)}[what]
    changed = []

    def unpack(t):
        if not ours(t):
            return t
        if t.dim() == 1:
            other = t.new_zeros((t.shape[0], 2))[:, 0].copy_(t)
        else:
            dims = (1, 2) if t.dtype == torch.bfloat16 else (-1, -2)          # (heads interleaved: still 16-byte rows)
            other = t.transpose(*dims).contiguous().transpose(*dims)
        changed.append(other.stride() != t.stride())
        return other

    want = torch.autograd.grad(sa.sparse_attention(*leaves, mask, 128, 32, mask_metadata=md), leaves, w)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach(), unpack):
        out = sa.sparse_attention(*leaves, mask, 128, 32, mask_metadata=md)
    got = torch.autograd.grad(out, leaves, w)
    assert any(changed)
    for name, g, r in zip(("dq", "dk", "dv"), got, want):
        assert torch.equal(g, r), name
