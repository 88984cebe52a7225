"""Scores that the first try of a step, against the row's present reference, does not fit: the reference moves to the
row's maximum and the step is done a second time.  Some rows, some tiles, every tile, the last one a CTA has, against the
generic kernel, which always keeps the running maximum; and rows whose result is known to the bit because their
reference must have moved."""
import math

import pytest
import torch

import sparseattention_b200 as sa

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(q, k, v, mask, bk):
    return sa.sparse_attention(q, k, v, mask, 128, bk, return_lse=True, check_status=True)


@pytest.mark.parametrize("D,bk", [(64, 32), (128, 64)])
@pytest.mark.parametrize("what", ["large", "small", "mixed", "one row", "large v", "empty rows"])
def test_tiles_that_need_a_maximum(native_lib, what, D, bk):
    B, H, S = 2, 41, 512                                       # 328 tiles: several per CTA, not a whole number of rounds
    g = torch.Generator(device=DEV).manual_seed(D + len(what))
    q, k, v = (torch.randn((B, H, S, D), generator=g, device=DEV) for _ in range(3))
    mask = (torch.rand((B, 1, S // 32, S // 32), generator=g, device=DEV) < 0.6).repeat_interleave(32, 2).repeat_interleave(32, 3)
    mask = mask & (torch.rand((B, 1, S, S), generator=g, device=DEV) < 0.9)
    mask[..., 0] = True
    if what == "large":                                        # every row's maximum far above the threshold
        q *= 12
    elif what == "small":                                      # every score near -200 in base 2: exp2 of it is 0
        q, k = q.abs() * 3, -k.abs() * 3 - 1
    elif what == "mixed":                                      # some heads, some blocks
        q[:, ::7] *= 14
        q[1, 3, 128:256] *= 20
    elif what == "one row":
        q[1, H - 1, S - 1] *= 25
    elif what == "large v":                                    # products with scores in the tens would overflow
        q *= 3.5
        v *= 2.0 ** 100
    else:
        q[:, ::5] *= 14
        mask[:, :, 100:140] = False
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    out, lse = _run(q, k, v, mask, bk)
    want, want_lse = sa.sparse_attention(q, k, v, mask, 128, bk, return_lse=True, impl="simt")
    # two results, each with P and the output rounded to bf16: 2 (2^-9 + 2^-9) of the largest |v|, 2^-10 of it on average
    vmax = v.float().abs().max().item()
    diff = (out.float() - want.float()).abs() / vmax
    assert torch.isfinite(out).all() and diff.max().item() <= 2.0 ** -7 and diff.mean().item() <= 2.0 ** -10
    live = mask.any(-1).expand(B, H, S)
    # scores of up to 2^10 in base 2: a few roundings (2^-24) in the scale, the maximum, the sum and the logarithm
    assert (lse - want_lse)[live].abs().max().item() <= 16 * 2.0 ** -24 * max(8.0, want_lse[live].abs().max().item() * math.log2(math.e))
    assert bool((lse[~live] == -math.inf).all()) and bool((out[~live.unsqueeze(-1).expand_as(out)] == 0).all())
    again, again_lse = _run(q, k, v, mask, bk)
    assert torch.equal(out, again) and torch.equal(lse, again_lse)
    part, _ = _run(q[:, 7:8], k[:, 7:8], v[:, 7:8], mask, bk)  # another schedule of the tiles: the same bits
    assert torch.equal(part, out[:, 7:8])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,Sq,Sk,D,bk,splits", [
    (2, 41, 512, 512, 128, 32, None),                          # several tiles per CTA
    (1, 3, 256, 512, 64, 128, 1),
    (1, 2, 128, 2048, 128, 64, 4),                             # one query block, its walk cut in four
    (2, 3, 160, 1024, 64, 32, None),                           # a short last query block
    (1, 2, 32, 4096, 128, 32, None),                           # nothing but a short block, the walk cut
])
def test_rows_with_one_far_key_return_its_value(native_lib, B, H, Sq, Sk, D, bk, splits, dtype):
    """A row that attends a single key whose score lies outside [-4, 8] takes that score as its reference: P is
    exp2 of a rounding error (1 in either 16-bit type), so the row of V comes back bit for bit.  P taken against
    another reference would be rounded (2^-9 in bf16) and the quotient with the fp32 sum with it."""
    g = torch.Generator(device=DEV).manual_seed(Sq + Sk + D)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    k, v = (rnd(B, H, Sk, D).to(dtype) for _ in range(2))
    at = torch.randint(0, Sk, (B, 1, Sq), generator=g, device=DEV)
    mask = torch.zeros((B, 1, Sq, Sk), dtype=torch.bool, device=DEV).scatter_(3, at[..., None], True)
    key = k.float().gather(2, at.expand(B, H, Sq)[..., None].expand(-1, -1, -1, D))
    x = torch.rand((B, H, Sq), generator=g, device=DEV) * 24 + 9.5          # log2 units
    x[..., 1::2] = 4 - x[..., 1::2]                                         # -5.5 ... -29.5
    scale = D ** -0.5 * math.log2(math.e)
    q = (key * (x / scale / key.square().sum(-1))[..., None]).to(dtype)
    out, lse = sa.sparse_attention(q, k, v, mask, 32 if Sq % 128 else 128, bk, return_lse=True, check_status=True, splits=splits)
    assert torch.equal(out, v.gather(2, at.expand(B, H, Sq)[..., None].expand(-1, -1, -1, D)))
    # q and k are exact 16-bit values, the product is summed in fp32: D roundings of at most |q||k| 2^-24, and the scale
    want = (q.double() * key.double()).sum(-1) * D ** -0.5
    bound = (D + 4) * 2.0 ** -24 * (q.double().abs() * key.double().abs()).sum(-1) * D ** -0.5
    assert bool(((lse.double() - want).abs() <= bound + 2.0 ** -22).all())


@pytest.mark.parametrize("D,bk", [(128, 32), (64, 128)])
def test_low_scores_keep_the_precision_of_small_values(native_lib, D, bk):
    """Every score near -46 in base 2 and V of 2^-106: P against 0 would make products of 2^-152, past the end of fp32;
    against the row's maximum nothing is lost.  Bound: P and the result rounded to bf16, 2^-9 each, of the largest |v|."""
    B, H, S = 1, 6, 512
    g = torch.Generator(device=DEV).manual_seed(D)
    q, k, v = (torch.randn((B, H, S, D), generator=g, device=DEV) for _ in range(3))
    c = math.sqrt(46 / (D ** -0.5 * math.log2(math.e)))
    q[..., 0], k[..., 0] = c, -c
    v *= 2.0 ** -106
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    mask = (torch.rand((B, 1, S, S), generator=g, device=DEV) < 0.7) | torch.eye(S, dtype=torch.bool, device=DEV)
    out = sa.sparse_attention(q, k, v, mask, 128, bk, check_status=True)
    x = (q.double() @ k.double().transpose(2, 3) * D ** -0.5).masked_fill(~mask, -math.inf)
    want = torch.softmax(x, -1) @ v.double()
    assert (out.double() - want).abs().max().item() <= 2.0 ** -8 * v.double().abs().max().item()
    assert ((out.double() - want).norm() / want.norm()).item() <= 2.0 ** -7
