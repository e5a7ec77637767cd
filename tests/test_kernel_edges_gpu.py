"""The kernels at the sizes where their tiling can go wrong, against the CPU restatement of the reference arithmetic.

Tolerance as in ``test_attn_gpu.py``: cosine similarity >= 0.999 and relative L1 <= 2e-2, LSE within 2e-3.
"""
import pytest
import torch

import sageattention_b200 as sa
from oracle import sage3
from tests import _util as U
from tests.test_attn_gpu import COS_MIN, REL_L1_MAX, oracle_on_device_operands

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one and two key tiles, a last key tile of one key, query tiles without a partner, query tiles that see no key or one
# key tile while their partner sees more, heads whose work items land on several rounds of the persistent grid
@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,D,causal", [
    (1, 2, 2, 1, 129, 128, False), (1, 2, 1, 129, 1, 64, False), (1, 4, 2, 257, 383, 128, True), (1, 4, 4, 640, 130, 128, True),
    (1, 4, 4, 511, 129, 64, True), (3, 60, 20, 129, 128, 128, True), (3, 60, 20, 385, 257, 64, False)])
def test_attention_at_tile_edges(B, Hq, Hkv, Nq, Nk, D, causal):
    q, k, v = U.make_qkv(B, Hq, Hkv, Nq, Nk, D, seed=Nq + Nk + D, device=DEV)
    z = sa.quantize_qkv(q, k, v)
    out, lse = sa.fp4_attention(z, is_causal=causal, return_lse=True, check_status=True)
    want, want_lse = oracle_on_device_operands(z, D ** -0.5, causal, return_lse=True)
    cos, l1 = sage3.accuracy(out.float().cpu(), want.to(torch.bfloat16).float())
    assert torch.isfinite(out).all() and cos >= COS_MIN and l1 <= REL_L1_MAX, (cos, l1)
    fin = torch.isfinite(want_lse)
    assert torch.allclose(lse.cpu()[fin], want_lse[fin], atol=2e-3, rtol=1e-4)
    assert bool(torch.isneginf(lse.cpu()[~fin]).all())


# K means added up from partial sums in the K kernel, which takes the query blocks of a whole GQA group as one list of rows:
# one row, 128 and 129 of them, sums of one chunk of tokens and of many, a head dim with channels to fill up
@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,D", [
    (1, 8, 2, 1, 300, 128), (2, 8, 8, 16384, 129, 64), (1, 4, 1, 32 * 128 + 1, 257, 128), (1, 12, 2, 300, 20000, 64), (1, 4, 2, 260, 511, 96)])
def test_k_means_and_delta_s_of_the_operator(B, Hq, Hkv, Nq, Nk, D):
    q, k, v = U.make_qkv(B, Hq, Hkv, Nq, Nk, 128 if D == 96 else D, seed=Nq + Nk, device=DEV)
    if D == 96:
        out = sa.sageattn(q[..., :96], k[..., :96], v[..., :96], sm_scale=0.1, check_status=True)
        want = sa.sageattn(*(torch.nn.functional.pad(t[..., :96], (0, 32)) for t in (q, k, v)), sm_scale=0.1)[..., :96]
        assert torch.equal(out, want)
        return
    z = sa.quantize_qkv(q, k, v)
    ref_km = k.float().mean(dim=2).to(torch.bfloat16).float()
    assert ((z.km.float() - ref_km).abs() <= ref_km.abs() * 2.0 ** -7 + 1e-3).all()
    ks = (k.float() - z.km.float()[:, :, None]).to(torch.bfloat16).float().repeat_interleave(Hq // Hkv, dim=1)
    want = torch.matmul(z.qm.float(), ks.transpose(-1, -2))
    assert torch.allclose(z.delta_s[..., :Nk].float(), want, atol=2e-2 * float(want.abs().max()), rtol=1e-2)
    assert (z.delta_s[..., Nk:] == 0).all()
    assert torch.equal(sa.sageattn(q, k, v, check_status=True), sa.fp4_attention(z))


# the work order of variable-length batches: more entries than threads and than SMs, sequences of no and one query, one
# tile, two and three; and one sequence alone
@pytest.mark.parametrize("n,causal,D", [(300, True, 128), (300, False, 64), (1, True, 64)])
def test_varlen_work_order_reaches_every_query_tile(n, causal, D):
    lens = [(0, 1, 128, 129, 256, 257, 385)[(5 * i + 3) % 7] for i in range(n)]
    g = torch.Generator().manual_seed(n)
    q, k, v = (torch.randn(sum(lens), h, D, generator=g).to(torch.bfloat16).to(DEV) for h in (4, 2, 2))
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    out = sa.sageattn_varlen(q, k, v, cu, cu, max(lens), max(lens), is_causal=causal, check_status=True)
    for i in range(n):
        s = slice(int(cu[i]), int(cu[i + 1]))
        if lens[i] > 0 and (i < 14 or i > n - 8):
            one = sa.sageattn(q[s][None], k[s][None], v[s][None], tensor_layout="NHD", is_causal=causal)[0]
            cos, l1 = sage3.accuracy(out[s].float().cpu(), one.float().cpu())
            assert cos >= 0.9995 and l1 <= 2e-2, (i, lens[i], cos, l1)
    assert torch.isfinite(out).all() and (out.float().abs().amax(dim=(1, 2)) > 0).all()


# the K-packing operator packs on the way into the quantisers: bit for bit what pack_kv + quantize_qkv + fp4_attention give;
# part of a group, one group, a whole tile of groups and one token more, several rounds of query blocks in the K kernel
@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,D,causal,pbm,layout", [
    (1, 2, 2, 40, 1, 128, False, True, "HND"), (2, 4, 2, 130, 15, 64, False, False, "NHD"), (1, 4, 2, 300, 120, 128, True, True, "HND"),
    (2, 2, 2, 257, 121, 64, True, False, "HND"), (1, 8, 1, 2200, 2200, 128, True, True, "NHD"), (1, 8, 1, 2200, 1000, 64, False, False, "NHD")])
def test_packing_operator_equals_its_parts(B, Hq, Hkv, Nq, Nk, D, causal, pbm, layout):
    q, k, v = U.make_qkv(B, Hq, Hkv, Nq, Nk, D, seed=Nq + Nk, layout=layout, device=DEV)
    got = sa.sageattn4_blackwell(q, k, v, tensor_layout=layout, is_causal=causal, per_block_mean=pbm, check_status=True)
    kp, vp, lam, _ = sa.pack_kv(k, v, layout, split_first=not pbm)
    if layout == "NHD":
        kp, vp = kp.transpose(1, 2), vp.transpose(1, 2)
    z = sa.quantize_qkv(q, kp, vp, layout, per_block_mean=pbm, smooth_k=False)
    z.k_lambda, z.mean_slot_first, z.nk_slots = lam, not pbm, sa._lib.load().sage3_packed_len(Nk)
    assert torch.equal(got, sa.fp4_attention(z, is_causal=causal, tensor_layout=layout))


# up to one query tile per SM: items of one tile, of a list that runs over the heads of a GQA group; and the sizes around that
# many, causal or not
@pytest.mark.parametrize("B,Hq,Hkv,Nq,D,causal", [
    (1, 148, 37, 100, 64, True), (1, 149, 149, 128, 64, False), (2, 37, 37, 200, 128, True), (1, 6, 2, 385, 128, False)])
def test_one_query_tile_per_item(B, Hq, Hkv, Nq, D, causal):
    q, k, v = U.make_qkv(B, Hq, Hkv, Nq, 300, D, seed=Nq + Hq, device=DEV)
    z = sa.quantize_qkv(q, k, v)
    out, lse = sa.fp4_attention(z, is_causal=causal, return_lse=True, check_status=True)
    want, want_lse = oracle_on_device_operands(z, D ** -0.5, causal, return_lse=True)
    cos, l1 = sage3.accuracy(out.float().cpu(), want.to(torch.bfloat16).float())
    assert torch.isfinite(out).all() and cos >= COS_MIN and l1 <= REL_L1_MAX, (cos, l1)
    fin = torch.isfinite(want_lse)
    assert torch.allclose(lse.cpu()[fin], want_lse[fin], atol=2e-3, rtol=1e-4)


# a key whose scores are NaN (K not smoothed, else every key is) at each place of a pair of 16-key blocks, of which some columns
# take another exponential than the others: rows that see it are zero with a NaN LSE, rows that do not are as without it.  Two
# tiles of query rows per item, one, packed sequences, and few query rows
@pytest.mark.parametrize("Nq,D,causal,op", [(300, 128, False, "dense"), (300, 64, True, "dense"), (100, 128, True, "dense"),
                                            (300, 64, False, "varlen"), (1, 128, False, "dense"), (4, 64, True, "dense")])
def test_nan_score_counts_alike_at_every_key(Nq, D, causal, op):
    H, Nk = 64, 600
    q, k, v = U.make_qkv(1, H, H, Nq, Nk, D, seed=Nq + D, k_offset_std=0.0, device=DEV)

    def run(k):
        if op == "dense":
            return sa.sageattn3_blackwell(q, k, v, is_causal=causal, smooth_k=False, return_lse=True, check_status=True)
        cu = [torch.tensor([0, n], dtype=torch.int32, device=DEV) for n in (Nq, Nk)]
        rows = [t[0].transpose(0, 1).contiguous() for t in (q, k, v)]
        return sa.sageattn_varlen(*rows, *cu, Nq, Nk, is_causal=causal, smooth_k=False, check_status=True).transpose(0, 1)[None], None

    want, want_lse = run(k)
    key = Nk - 330 + torch.arange(H, device=DEV) + 128 * (torch.arange(H, device=DEV) % 2)
    bad = k.clone()
    bad[0, torch.arange(H, device=DEV), key, 5] = float("nan")
    out, lse = run(bad)
    last = torch.arange(Nq, device=DEV) + Nk - Nq if causal else torch.full((Nq,), Nk, device=DEV)   # last visible key
    sees = last[None] >= key[:, None]
    assert bool(sees.any()) and (Nq < 300 or not causal or not bool(sees.all()))
    assert bool((out[0][sees] == 0).all()), sorted({int(h) % 32 for h in (out[0] != 0).any(-1).logical_and(sees).any(-1).nonzero()})
    assert torch.equal(out[0][~sees], want[0][~sees])
    if lse is not None:
        assert bool(torch.isnan(lse[0][sees]).all()) and torch.equal(lse[0][~sees], want_lse[0][~sees])


# as many query tiles as CTAs with a margin, one more and one fewer (items of one or of two tiles), and few query rows per head,
# whose kernels have no margin: the same bits
@pytest.mark.parametrize("Hq,Hkv,Nq,margin", [(100, 100, 128, 47), (100, 100, 128, 48), (100, 100, 128, 49), (35, 7, 300, 43), (35, 7, 300, 44), (8, 2, 1, 100)])
def test_sm_margin_around_one_query_tile_per_cta(Hq, Hkv, Nq, margin):
    q, k, v = U.make_qkv(1, Hq, Hkv, Nq, 500, 128, seed=Hq + Nq, device=DEV)
    want = sa.sageattn(q, k, v, is_causal=True)
    assert torch.equal(sa.sageattn(q, k, v, is_causal=True, sm_margin=margin, check_status=True), want)


# K channel sums first or last (8 to 96 MB of K, counted with the longest sequence's length) in the first launch; sequences
# without keys among them
@pytest.mark.parametrize("lens", [[8000] + [120, 0, 121] * 36, [2000] * 8 + [500], [100, 0, 3000]])
def test_varlen_k_sums_first_and_last(lens):
    g = torch.Generator().manual_seed(len(lens))
    q, k, v = (torch.randn(sum(lens), h, 128, generator=g).to(torch.bfloat16).to(DEV) for h in (2, 2, 2))
    k += 2.0 * torch.randn(1, 2, 128, generator=g).to(torch.bfloat16).to(DEV)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    out = sa.sageattn_varlen(q, k, v, cu, cu, max(lens), max(lens), is_causal=True, check_status=True)
    for i in range(len(lens)):
        s = slice(int(cu[i]), int(cu[i + 1]))
        if lens[i] > 0 and (i < 8 or i > len(lens) - 4):
            one = sa.sageattn(q[s][None], k[s][None], v[s][None], tensor_layout="NHD", is_causal=True)[0]
            cos, l1 = sage3.accuracy(out[s].float().cpu(), one.float().cpu())
            assert cos >= 0.9995 and l1 <= 2e-2, (i, lens[i], cos, l1)
    assert torch.isfinite(out).all()
