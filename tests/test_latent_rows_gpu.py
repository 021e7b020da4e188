"""What a decode step of few rows of a latent mixer runs on: the launch that makes its queries' rows and the cache's, the per-head
product of few rows, and the norm with a row in a block's registers; each against the kernels of any number of rows or 64 bits."""
import pytest
import torch

from rosellm_b200.ops import kernels as K
from rosellm_b200.parts.standard import rotary_frequencies

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ints(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# heads fewer and more than tokens, latents that end inside a slice of 64, rotated parts with entries that are not turned, none, and
# rows filled up with zeros
@pytest.mark.parametrize("rows", [1, 9, 16])
@pytest.mark.parametrize("heads,plain,rank,rot,dims", [(16, 128, 512, 64, 64), (3, 64, 72, 8, 4), (2, 256, 40, 0, 0), (20, 64, 100, 20, 20)])
def test_prepare(rows, heads, plain, rank, rot, dims):
    g = torch.Generator(device=DEV).manual_seed(rows + rank)
    width, page, head_in = -(-(rank + rot) // 8) * 8, 8, -(-(plain + rot) // 8) * 8
    q = torch.randn(rows, heads * head_in, generator=g, device=DEV).bfloat16()
    uk = (torch.randn(heads, rank, plain, generator=g, device=DEV) * plain ** -0.5).bfloat16()
    dkv = torch.randn(rows, rank + rot + 3, generator=g, device=DEV)
    gamma = 1 + 0.1 * torch.randn(rank, generator=g, device=DEV)
    positions, req = _ints([37 * i for i in range(rows)]), _ints(list(range(rows)))
    slots = _ints([rows - 1 - i if i != 2 else -1 for i in range(rows)])  # the third row is padding
    table = torch.arange(rows * 80, dtype=torch.int32, device=DEV).view(rows, 80)
    freq = rotary_frequencies(max(dims, 2), 300.0).to(DEV)
    pools = [torch.full((rows * 80, 1, 1, page, width), 7.0, device=DEV).bfloat16() for _ in range(2)]
    out = [torch.full((rows, heads * width), float("nan"), device=DEV).bfloat16() for _ in range(2)]
    where = dict(rank=rank, rot_dim=rot, rot_mult=1.25)
    assert K.latent_prepare_possible(rows, plain, head_in, torch.bfloat16)
    K.latent_prepare(q, uk, out[0], freq, positions, n_heads=heads, head_in=head_in, plain=plain, rot_dims=dims, row_width=width, dkv=dkv,
                     gamma=gamma, eps=1e-5, pool=pools[0], block_table=table, req_of_token=req, slots=slots, max_pos=80 * page, **where)
    K.latent_kv_write(dkv, gamma, 1e-5, freq, dims, pools[1], table, positions, req, slots, max_pos=80 * page, **where)
    K.latent_q_rope(q, out[1], freq, positions, n_heads=heads, head_in=head_in, plain=plain, rot_dims=dims, row_width=width, **where)
    want = torch.einsum("thp,hrp->thr", q.view(rows, heads, head_in)[..., :plain].double(), uk.double())
    got = [o.view(rows, heads, width) for o in out]
    assert torch.equal(got[0][..., rank:], got[1][..., rank:])  # the rotation: the same arithmetic
    # a bfloat16 rounding, and float32 sums of products of order 1
    assert ((got[0][..., :rank].double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()
    # the norm's sum in another order: at most a step of bfloat16 apart
    a, b = pools[0].double(), pools[1].double()
    assert ((a - b).abs() <= b.abs() * 2.0 ** -7).all() and (a[..., rank:] == b[..., rank:]).all()
    # without rows of the cache
    again = torch.empty_like(out[0])
    K.latent_prepare(q, uk, again, freq, positions, n_heads=heads, head_in=head_in, plain=plain, rot_dims=dims, row_width=width, **where)
    assert torch.equal(again, out[0])
    K.check_status(torch.device(DEV))


def test_prepare_flags_a_missing_page_and_a_position_beyond():
    q, uk, out = torch.zeros(2, 72, device=DEV).bfloat16(), torch.zeros(1, 8, 64, device=DEV).bfloat16(), torch.zeros(2, 8, device=DEV).bfloat16()
    for table, positions, bit in ([[-1], [-1]], [0, 0], 4), ([[0], [1]], [0, 99], 2):
        K.latent_prepare(q, uk, out, None, _ints(positions), n_heads=1, head_in=72, plain=64, rank=8, rot_dim=0, rot_dims=0, row_width=8,
                         dkv=torch.zeros(2, 8, device=DEV), gamma=torch.ones(8, device=DEV), eps=1e-5,
                         pool=torch.zeros(2, 1, 1, 8, 8, device=DEV).bfloat16(), block_table=_ints(table), req_of_token=_ints([0, 1]),
                         slots=_ints([0, 1]), max_pos=8)
        torch.cuda.synchronize()
        status = K.status_word(torch.device(DEV))
        assert int(status.item()) == bit
        status.zero_()


# one to eight warps along K, one to four blocks of 64 elements a warp; columns that end inside a warp's eight; a gate
@pytest.mark.parametrize("rows", [1, 8, 9, 16])
@pytest.mark.parametrize("k,n", [(64, 8), (128, 513), (256, 40), (512, 128), (1024, 17), (2048, 130), (192, 24)])
def test_head_product_of_few_rows(rows, k, n):
    g = torch.Generator(device=DEV).manual_seed(rows + k + n)
    heads = 3
    x = torch.randn(rows, heads, k + 8, generator=g, device=DEV).bfloat16()
    w = (torch.randn(heads, n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    gate = torch.randn(rows, heads * n, generator=g, device=DEV)
    want = torch.einsum("thk,hnk->thn", x[..., :k].double(), w.double())
    for with_gate in (False, True):
        out = torch.full((rows, heads, n + 4), 5.0, device=DEV).bfloat16()
        K.head_linear(x, w, out, n_tokens=rows, n_heads=heads, k=k, n=n, in_strides=(heads * (k + 8), k + 8), w_strides=(k * n, 1, k),
                      out_strides=(heads * (n + 4), n + 4), gate=gate if with_gate else None, gate_strides=(heads * n, n, 1))
        ref = want * torch.sigmoid(gate.double()).view(rows, heads, n) if with_gate else want
        assert ((out[..., :n].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all() and (out[..., n:] == 5.0).all()


@pytest.mark.parametrize("width", [768, 1020, 1024, 1028, 2048, 4096, 4100])
def test_norm_added_with_the_row_in_registers(width):
    """Beside a row that is no whole number of 16-byte pieces of its stride, which the kernel that reads twice takes."""
    g = torch.Generator(device=DEV).manual_seed(width)
    y, gamma = torch.randn(5, width, generator=g, device=DEV), torch.randn(width, generator=g, device=DEV)
    base = torch.randn(5, width, generator=g, device=DEV)
    x, copy = base.clone(), torch.empty(5, width, device=DEV).bfloat16()
    K.rmsnorm_add(y, gamma, 1e-5, x, 0.5, copy)
    want = base.double() + 0.5 * y.double() / torch.sqrt((y.double() ** 2).mean(-1, keepdim=True) + 1e-5) * gamma.double()
    assert ((x.double() - want).abs() <= 4e-6 * (1 + want.abs())).all() and torch.equal(copy, x.bfloat16())
    wide = torch.empty(5, width + 1, device=DEV)
    wide[:, :width] = base
    K.rmsnorm_add(y, gamma, 1e-5, wide[:, :width], 0.5, None)
    assert ((wide[:, :width] - x).abs() <= 4e-6 * (1 + x.abs())).all()


# one warp's rows in four warps and in eight, two warps' rows, four's; latents that end inside a slice and rows that end inside a step of
# 32; pages of a power of two and of 24; requests of one key, of part of a tile of keys, of whole tiles, of parts without a key
@pytest.mark.parametrize("splits", [1, 2, 3, 8, 9])  # whole, in clusters, more parts than a cluster takes
@pytest.mark.parametrize("heads,rank,rot,page", [(16, 512, 64, 16), (3, 40, 8, 24), (16, 100, 20, 8), (5, 200, 8, 24), (20, 512, 40, 16), (40, 128, 24, 16)])
def test_decoded_tokens_in_parts(heads, rank, rot, page, splits):
    lens, width = [1, 31, 33, 64, 200, 371], rank + rot
    n, width = len(lens), width + (-width) % 8
    g = torch.Generator(device=DEV).manual_seed(heads * 7 + rank)
    per = -(-max(lens) // page)
    table = torch.randperm(n * per, generator=g, device=DEV).int().view(n, per).contiguous()
    pool = torch.randn(n * per, 1, 1, page, width, generator=g, device=DEV).bfloat16()
    q = torch.randn(n, heads * width, generator=g, device=DEV).bfloat16()
    sink, scale = torch.randn(heads, generator=g, device=DEV), width ** -0.5
    out = torch.full((n, heads * rank), float("nan"), device=DEV).bfloat16()
    ids, scratch = _ints(list(range(n))), [torch.empty(n * heads * splits, w, device=DEV) for w in (rank, 2)]
    K.latent_attention(q, pool, table, _ints(list(range(n + 1))), _ints(lens), ids, out, sink=sink, n_heads=heads, rank=rank, scale=scale,
                       tiles=None, n_tiles=0, decode_reqs=ids, n_decode=n, decode_by_request=True, n_splits=splits, part_o=scratch[0],
                       part_ml=scratch[1])
    K.check_status(torch.device(DEV))
    for r, length in enumerate(lens):
        rows = pool[table[r].long()].view(-1, width)[:length].double()
        scores = q[r].view(heads, width).double() @ rows.T * scale
        p = torch.softmax(torch.cat([scores, sink.double()[:, None]], 1), 1)[:, :-1]
        want, most = p @ rows[:, :rank], p @ rows[:, :rank].abs()
        # probabilities and the result each rounded to bfloat16, the parts' maxima apart from the whole's
        assert ((out[r].view(heads, rank).double() - want).abs() <= 2.0 ** -8 * (want.abs() + 1.5 * most) + 1e-5).all()


# whole pairs of columns and an odd last one, a stride between heads that is odd: two columns stored together or each by itself
@pytest.mark.parametrize("n,gap", [(40, 0), (41, 0), (40, 3)])
def test_head_product_of_many_rows(n, gap):
    t, h, k = 37, 3, 72
    g = torch.Generator(device=DEV).manual_seed(n + gap)
    x = torch.randn(t, h * k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(h, k, n, generator=g, device=DEV) * k ** -0.5).bfloat16()
    out = torch.full((t, h, n + gap), 5.0, device=DEV).bfloat16()
    K.head_linear(x, w, out, n_tokens=t, n_heads=h, k=k, n=n, in_strides=(h * k, k), w_strides=(k * n, n, 1),
                  out_strides=(h * (n + gap), n + gap))
    want = torch.einsum("thk,hkn->thn", x.view(t, h, k).double(), w.double())
    # a bfloat16 rounding, and float32 sums of products of order 1
    assert ((out[..., :n].double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()
    assert (out[..., n:] == 5.0).all()
