"""The causal prefill kernel over the paged cache against fp32 torch attention on the contiguous history.

Each case: sequences with some history already in their pages receive a chunk of new tokens
(ktk_append_tokens), then ktk_prefill_attention attends every new token to its own prefix.  Reference:
softmax(q K^T / sqrt(D)) V in fp32 with the causal mask over absolute positions -- what
flashinfer.single_prefill_with_kv_cache(causal=True) computes in LiteSys/litesys/attention/batch_cache.py:129-145.
"""
import math

import pytest
import torch

from helpers import paged_state, to_dev

pytestmark = pytest.mark.gpu


def _reference(q, k, v, G):
    """q [n_new, Hq, D], k/v [Hkv, total, D] fp32; new tokens are the last n_new positions."""
    n_new, Hq, D = q.shape
    total = k.shape[1]
    pos = torch.arange(total - n_new, total, device=q.device)
    mask = torch.arange(total, device=q.device)[None, :] <= pos[:, None]              # [n_new, total]
    kk = k.repeat_interleave(G, dim=0)                                                 # [Hq, total, D]
    vv = v.repeat_interleave(G, dim=0)
    logits = torch.einsum("nhd,htd->hnt", q, kk) / math.sqrt(D)
    logits = logits.masked_fill(~mask[None], float("-inf"))
    return torch.einsum("hnt,htd->nhd", torch.softmax(logits, dim=-1), vv)


@pytest.mark.parametrize("dtype,variant", [(torch.bfloat16, 0), (torch.bfloat16, 1), (torch.bfloat16, 2), (torch.bfloat16, 3),
                                           (torch.float32, 0)])
@pytest.mark.parametrize("G,Hkv,sink", [(4, 2, 0), (8, 1, 4), (2, 2, 4), (1, 3, 0)])
def test_prefill_matches_causal_attention(cuda_device, dtype, variant, G, Hkv, sink):
    from kinetics_b200 import ops
    # (history, new tokens): a fresh prompt, a chunk behind a long history, a chunk ending on a page edge, a
    # single new token, a prompt shorter than the sink, an empty chunk
    hist = [0, 300, 16 * 7 - 5 + sink, 77, 0, 40]
    new = [137, 61, 5, 1, 3, 0]
    B = len(hist)
    lens = [h + n for h, n in zip(hist, new)]
    g = torch.Generator().manual_seed(17 + G + sink)
    L = max(lens)
    k = torch.randn(B, Hkv, L, 128, generator=g).to(dtype).float()
    v = torch.randn(B, Hkv, L, 128, generator=g).to(dtype).float()
    # the pages hold only the history at first; the kernel under test's companion writes the chunk
    st = paged_state(k, v, lens, dtype, seed=3, sink=sink, fill=0.0)
    d = to_dev(st, cuda_device)
    status = ops.new_status(cuda_device)
    q_indptr = torch.tensor([sum(new[:i]) for i in range(B + 1)], dtype=torch.int32, device=cuda_device)
    total_new = sum(new)
    q = torch.randn(total_new, Hkv * G, 128, generator=g).to(dtype).to(cuda_device)
    view = ops.PageView(sink_tokens=sink, local_tokens=1) if sink else None
    # write the chunks again through the append kernel (the fixture already holds them: same bytes)
    k_new = torch.cat([k[b, :, hist[b]:lens[b]].transpose(0, 1) for b in range(B)]).to(dtype).to(cuda_device)
    v_new = torch.cat([v[b, :, hist[b]:lens[b]].transpose(0, 1) for b in range(B)]).to(dtype).to(cuda_device)
    before = d["kv_cache"].clone()
    ops.append_tokens(k_new.contiguous(), v_new.contiguous(), q_indptr, d["kv_cache"], None, d["kv_indices"],
                      d["kv_indptr"], d["kv_last_page_len"], status=status, view=view)
    assert torch.equal(before, d["kv_cache"])
    out = ops.prefill_attention(q, q_indptr, max(new), d["kv_cache"], d["kv_indices"], d["kv_indptr"],
                                d["kv_last_page_len"], variant=variant, status=status, view=view)
    ops.raise_on_status(status)
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    for b in range(B):
        if new[b] == 0:
            continue
        lo, hi = int(q_indptr[b]), int(q_indptr[b + 1])
        ref = _reference(q[lo:hi].float(), k[b, :, :lens[b]].to(cuda_device), v[b, :, :lens[b]].to(cuda_device), G)
        torch.testing.assert_close(out[lo:hi].float(), ref, rtol=tol, atol=tol)


def test_prefill_long_prompt_many_sequences(cuda_device):
    # several 2000-token prompts in one launch, G = 4: tiles of 8 tokens, 126 pages for the last tile
    from kinetics_b200 import ops
    B, Hkv, G, n = 3, 2, 4, 2003
    g = torch.Generator().manual_seed(5)
    k = torch.randn(B, Hkv, n, 128, generator=g).to(torch.bfloat16).float()
    v = torch.randn(B, Hkv, n, 128, generator=g).to(torch.bfloat16).float()
    st = paged_state(k, v, [n] * B, torch.bfloat16, seed=4, fill=0.0)
    d = to_dev(st, cuda_device)
    q_indptr = torch.arange(B + 1, dtype=torch.int32, device=cuda_device) * n
    q = torch.randn(B * n, Hkv * G, 128, generator=g).to(torch.bfloat16).to(cuda_device)
    status = ops.new_status(cuda_device)
    out = ops.prefill_attention(q, q_indptr, n, d["kv_cache"], d["kv_indices"], d["kv_indptr"], d["kv_last_page_len"],
                                status=status)
    rows = ops.prefill_attention(q, q_indptr, n, d["kv_cache"], d["kv_indices"], d["kv_indptr"], d["kv_last_page_len"],
                                 variant=1, status=status)
    ops.raise_on_status(status)
    torch.testing.assert_close(out.float(), rows.float(), rtol=2e-2, atol=2e-2)
    ref = _reference(q[n:2 * n].float(), k[1].to(cuda_device), v[1].to(cuda_device), G)
    torch.testing.assert_close(out[n:2 * n].float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("G,Hkv,sink,B", [(8, 4, 0, 7), (8, 4, 4, 7), (4, 6, 0, 32), (4, 1, 0, 32), (8, 1, 4, 16), (2, 3, 0, 33)])
def test_prefill_of_unequal_sequences_over_more_than_one_round(cuda_device, G, Hkv, sink, B):
    """Portions of very different lengths behind very different histories, some empty: the CTAs take them by length (up to 32
    sequences in one to two and a half rounds of CTAs).  Every row is written once, with what the row-by-row kernel gives.  Bound: as in the other prompts."""
    from kinetics_b200 import ops
    new = ([700, 3, 0, 450, 64, 65, 1200] * 5)[:B]
    hist = ([100, 2500, 40, 0, 900, 10, 5] * 5)[:B]
    lens = [h + n for h, n in zip(hist, new)]
    g = torch.Generator().manual_seed(B)
    pages = [1 + max(0, -(-(n - sink) // 16)) if sink else -(-n // 16) for n in lens]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda_device)
    indptr, q_indptr = i32([sum(pages[:i]) for i in range(B + 1)]), i32([sum(new[:i]) for i in range(B + 1)])
    last = i32([(n - sink - 1) % 16 + 1 if sink and n > sink else n if sink else (n - 1) % 16 + 1 for n in lens])
    table = torch.randperm(sum(pages), generator=g).to(torch.int32).to(cuda_device)
    cache = torch.randn(sum(pages), 2, 16, Hkv, 128, generator=g).to(torch.bfloat16).to(cuda_device)
    q = torch.randn(sum(new), Hkv * G, 128, generator=g).to(torch.bfloat16).to(cuda_device)
    view, status = ops.PageView(sink_tokens=sink, local_tokens=1) if sink else None, ops.new_status(cuda_device)
    run = lambda variant: ops.prefill_attention(q, q_indptr, max(new), cache, table, indptr, last, variant=variant, status=status,
                                                view=view, out=torch.full_like(q, float("nan")))
    got, want = run(0), run(1)
    ops.raise_on_status(status)
    torch.testing.assert_close(got.float(), want.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("variant", [0, 2])
@pytest.mark.parametrize("G,sink", [(4, 0), (2, 4), (8, 4)])
def test_prefill_on_block_and_tile_edges(cuda_device, variant, G, sink):
    """Histories and chunks that end exactly on the edges the kernels cut at: 16-token pages, the 64-key blocks
    and the 128 / G-token tiles of the tcgen05 kernel (and one token to either side of them)."""
    from kinetics_b200 import ops
    Hkv = 2
    tile = 128 // G
    hist = [0, 64 - sink, 64, 128 + sink, 63, 0, 16 * 9]
    new = [tile, tile, 2 * tile, tile + 1, 1, 64 + sink + 1, tile - 1]
    B = len(hist)
    lens = [h + n for h, n in zip(hist, new)]
    g = torch.Generator().manual_seed(40 + G + sink)
    L = max(lens)
    k = torch.randn(B, Hkv, L, 128, generator=g).to(torch.bfloat16).float()
    v = torch.randn(B, Hkv, L, 128, generator=g).to(torch.bfloat16).float()
    st = paged_state(k, v, lens, torch.bfloat16, seed=9, sink=sink)           # unused slots hold NaN
    d = to_dev(st, cuda_device)
    status = ops.new_status(cuda_device)
    q_indptr = torch.tensor([sum(new[:i]) for i in range(B + 1)], dtype=torch.int32, device=cuda_device)
    q = torch.randn(sum(new), Hkv * G, 128, generator=g).to(torch.bfloat16).to(cuda_device)
    view = ops.PageView(sink_tokens=sink, local_tokens=1) if sink else None
    out = ops.prefill_attention(q, q_indptr, max(new), d["kv_cache"], d["kv_indices"], d["kv_indptr"],
                                d["kv_last_page_len"], variant=variant, status=status, view=view)
    ops.raise_on_status(status)
    assert torch.isfinite(out.float()).all()
    for b in range(B):
        lo, hi = int(q_indptr[b]), int(q_indptr[b + 1])
        ref = _reference(q[lo:hi].float(), k[b, :, :lens[b]].to(cuda_device), v[b, :, :lens[b]].to(cuda_device), G)
        torch.testing.assert_close(out[lo:hi].float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("G,sink,grow,n", [(4, 0, (0.1, 40.0, 200.0), 200), (1, 4, (1.0, 1.0, 90.0), 200), (2, 0, (60.0, 0.1, 30.0), 200),
                                           (8, 4, (0.1, 40.0, 200.0), 1300)])
def test_prefill_scores_that_outgrow_their_reference(cuda_device, G, sink, grow, n):
    """The exponentials' reference is the first block's maximum until a half block's sum passes 2^8: scores that grow by far
    more in the first half of a block of 128 keys, in its second half, in the block of the row itself; and that shrink.

    Bound: operands are the reference's own bf16 values, products of 128 columns are summed in fp32, so a score of up to about
    1000 is off by a few 1e-4, a weight by that share; bf16 weights add 2^-9 of each value: 2e-2, as in the other cases."""
    from kinetics_b200 import ops
    Hkv, hist = 2, 330                                       # the last case: more tiles than SMs, two to a CTA
    total = hist + n
    g = torch.Generator().manual_seed(7 + G)
    factor = torch.full((total,), grow[0])
    factor[140:170] = grow[1]                                # first half of the second block
    factor[230:236] = grow[2]                                # second half of it
    factor[hist + 20:hist + 90] = grow[2]                    # among the new tokens
    k = (torch.randn(1, Hkv, total, 128, generator=g) * factor[:, None]).to(torch.bfloat16).float()
    v = torch.randn(1, Hkv, total, 128, generator=g).to(torch.bfloat16).float()
    d = to_dev(paged_state(k, v, [total], torch.bfloat16, seed=3, sink=sink), cuda_device)
    q = torch.randn(n, Hkv * G, 128, generator=g).to(torch.bfloat16).to(cuda_device)
    q_indptr = torch.tensor([0, n], dtype=torch.int32, device=cuda_device)
    status = ops.new_status(cuda_device)
    view = ops.PageView(sink_tokens=sink, local_tokens=1) if sink else None
    out = ops.prefill_attention(q, q_indptr, n, d["kv_cache"], d["kv_indices"], d["kv_indptr"], d["kv_last_page_len"],
                                status=status, view=view)
    ops.raise_on_status(status)
    ref = _reference(q.float(), k[0].to(cuda_device), v[0].to(cuda_device), G)
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-2)


def _attend_exponents(dev, exponents, v, n, G=4):
    """Attention of the last n tokens over keys whose weights are 2^exponent for every query: q = (1, 2^-8, 0, ..), k = (whole
    part, 256 times the rest, 0, ..), both exact in bf16; sm_scale = ln 2."""
    from kinetics_b200 import ops
    e = torch.tensor(exponents)
    k = torch.zeros(1, 1, len(exponents), 128)
    k[0, 0, :, 0], k[0, 0, :, 1] = e.floor(), (e - e.floor()) * 256
    assert torch.equal(k.to(torch.bfloat16).float(), k)
    d = to_dev(paged_state(k, v, [len(exponents)], torch.bfloat16, seed=3), dev)
    q = torch.zeros(n, G, 128, dtype=torch.bfloat16, device=dev)
    q[..., 0], q[..., 1] = 1.0, 2.0 ** -8
    status = ops.new_status(dev)
    out = ops.prefill_attention(q, torch.tensor([0, n], dtype=torch.int32, device=dev), n, d["kv_cache"], d["kv_indices"],
                                d["kv_indptr"], d["kv_last_page_len"], sm_scale=math.log(2.0), status=status)
    ops.raise_on_status(status)
    return out.float().cpu()


#: 2^0.005615 = 1.0039: half way between two bf16 numbers, so that a weight of that mantissa is off by 2^-8 of itself in bf16
HALF_WAY = 1.4375 / 256


@pytest.mark.parametrize("at", [5, 100, 140, 200, 396])
def test_prefill_a_key_that_outweighs_all_others(cuda_device, at):
    """Its weight is 2^28 of the others': the row is its value, whose bf16 form the result is to the bit (400 others change it by
    less than 2^-19 of their size)."""
    exponents = [0.0] * 400
    exponents[at] = 28.0 + HALF_WAY
    v = torch.randn(1, 1, 400, 128, generator=torch.Generator().manual_seed(at)).to(torch.bfloat16).float()
    v += v.sign() * 0.5                                      # no value so small that the others matter in its last bit
    v = v.to(torch.bfloat16).float()
    out = _attend_exponents(cuda_device, exponents, v, 4)
    assert torch.equal(out, v[0, 0, at].expand_as(out))


def test_prefill_values_near_the_end_of_the_range(cuda_device):
    """Values of 2^104 behind scores that grow by 22: 8192 keys of weight 2^8 leave 2^107."""
    v = torch.full((1, 1, 400, 128), 2.0 ** 104)
    out = _attend_exponents(cuda_device, [0.0] * 150 + [22.0] * 100 + [0.0] * 150, v, 4)
    assert torch.equal(out, torch.full_like(out, 2.0 ** 104))


@pytest.mark.parametrize("G,tiles", [(1, 3), (4, 3), (8, 3), (4, 0), (8, 0)])
def test_prefill_rows_of_a_tile_are_free_of_later_values(cuda_device, G, tiles):
    """A value that is not finite spoils the rows that see its key, and may spoil those of their tile of 128 / G tokens before it,
    whose weight for it is 0.  Rows of the tiles in front stay what they are without it.  tiles 0: more than SMs, two to a CTA."""
    tile, tiles = 128 // G, tiles or torch.cuda.get_device_properties(cuda_device).multi_processor_count + 3
    n = tiles * tile
    v = torch.randn(1, 1, n, 128, generator=torch.Generator().manual_seed(G)).to(torch.bfloat16).float()
    clean = _attend_exponents(cuda_device, [0.0] * n, v, n, G)
    for at in (tile, tile + tile // 2, 2 * tile, n - tile - 1):
        spoilt = v.clone()
        spoilt[0, 0, at, ::2], spoilt[0, 0, at, 1::2] = float("inf"), float("nan")
        out = _attend_exponents(cuda_device, [0.0] * n, spoilt, n, G)
        ahead = at // tile * tile
        assert torch.equal(out[:ahead], clean[:ahead])
        assert not torch.isfinite(out[at:]).any()


@pytest.mark.parametrize("more", [-1, 0, 1, 17])
def test_prefill_with_about_as_many_tiles_as_sms(cuda_device, more):
    """A CTA takes one tile where all tiles find an SM, two otherwise: tiles of 16 tokens on either side of that, in one sequence
    and over several with an empty one.  Bound: as in the other cases."""
    from kinetics_b200 import ops
    G, tokens = 8, 16 * (torch.cuda.get_device_properties(cuda_device).multi_processor_count + more) - 3
    for new in ([tokens], [0, tokens // 2, 1, tokens - tokens // 2 - 1]):
        lens = [n + (5 if n else 0) for n in new]
        g = torch.Generator().manual_seed(tokens)
        k = torch.randn(len(new), 1, max(lens), 128, generator=g).to(torch.bfloat16).float()
        v = torch.randn(len(new), 1, max(lens), 128, generator=g).to(torch.bfloat16).float()
        d = to_dev(paged_state(k, v, lens, torch.bfloat16, seed=5), cuda_device)
        q = torch.randn(sum(new), G, 128, generator=g).to(torch.bfloat16).to(cuda_device)
        indptr = torch.tensor([sum(new[:i]) for i in range(len(new) + 1)], dtype=torch.int32, device=cuda_device)
        status = ops.new_status(cuda_device)
        out = ops.prefill_attention(q, indptr, max(new), d["kv_cache"], d["kv_indices"], d["kv_indptr"], d["kv_last_page_len"],
                                    status=status)
        ops.raise_on_status(status)
        for b, n in enumerate(new):
            lo = int(indptr[b])
            ref = _reference(q[lo:lo + n].float(), k[b, :, :lens[b]].to(cuda_device), v[b, :, :lens[b]].to(cuda_device), G)
            torch.testing.assert_close(out[lo:lo + n].float(), ref, rtol=2e-2, atol=2e-2)
