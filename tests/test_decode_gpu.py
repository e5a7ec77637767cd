"""Few query rows per head: the operator splits the keys over the chip there.  Against the CPU restatement of the reference
arithmetic, tolerance as in ``test_attn_gpu.py``: cosine similarity >= 0.999 and relative L1 <= 2e-2, LSE within 2e-3.
"""
import pytest
import torch

import sageattention_b200 as sa
from oracle import sage3
from tests import _util as U
from tests.test_attn_gpu import COS_MIN, REL_L1_MAX, oracle_on_device_operands

pytestmark = pytest.mark.gpu
DEV = "cuda"


# the fewest key tiles (and one fewer: the other kernel), a last tile of one key, key tiles that do not fill the runs, runs of
# several tiles; 1, 8, 9, 16 and 17 rows per kv head and the most there can be; causal rows that see the last keys or not
@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,D,causal", [
    (1, 2, 2, 1, 384, 128, False), (1, 2, 2, 1, 385, 128, False), (2, 4, 2, 4, 1023, 64, True), (1, 9, 1, 1, 1025, 64, False),
    (1, 2, 2, 8, 1153, 128, True), (1, 4, 1, 4, 2000, 128, True), (1, 17, 1, 1, 1000, 128, False), (1, 16, 2, 8, 1100, 64, True), (1, 4, 2, 16, 1025, 128, True),
    (1, 2, 1, 2, 33000, 128, True), (1, 2, 1, 1, 65537, 64, False), (40, 32, 8, 1, 1500, 128, False)])
def test_few_query_rows(B, Hq, Hkv, Nq, Nk, D, causal):
    q, k, v = U.make_qkv(B, Hq, Hkv, Nq, Nk, D, seed=Nq + Nk + D, device=DEV)
    out = sa.sageattn(q, k, v, is_causal=causal, check_status=True)
    out2, lse = sa.sageattn(q, k, v, is_causal=causal, return_lse=True, check_status=True)
    assert torch.allclose(out.float(), out2.float(), atol=2e-3, rtol=2e-2)
    z = sa.quantize_qkv(q, k, v)
    other, other_lse = sa.fp4_attention(z, is_causal=causal, return_lse=True)
    assert torch.isfinite(out).all()
    assert sage3.accuracy(out.float().cpu(), other.float().cpu())[1] <= 1e-3
    if B * Hq <= 64:
        want, want_lse = oracle_on_device_operands(z, D ** -0.5, causal, return_lse=True)
        cos, l1 = sage3.accuracy(out.float().cpu(), want.to(torch.bfloat16).float())
        assert cos >= COS_MIN and l1 <= REL_L1_MAX, (cos, l1)
    # (the kernel's own LSE lacks the K-mean term, which the operator adds)
    term = D ** -0.5 * torch.einsum("bhnd,bhd->bhn", q.float(), z.km.float().repeat_interleave(Hq // Hkv, dim=1))
    assert torch.allclose(lse, other_lse + term, atol=4e-3, rtol=1e-4)


# V quantised beside the scores: from 128 key tiles of all kv heads on (one fewer: beside the K sums), a last tile of one key, narrow
# rows, tokens strided; against the tile kernels on V quantised by its own launch, up to the order of fp32 sums (<= 1e-3, as above)
@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,d,layout", [
    (1, 1, 1, 1, 16256, 128, "HND"), (1, 1, 1, 1, 16257, 128, "HND"), (4, 8, 8, 1, 513, 72, "NHD"), (3, 32, 8, 2, 1000, 104, "HND"),
    (16, 8, 8, 8, 640, 128, "NHD")])
def test_v_quantised_beside_the_scores(B, Hq, Hkv, Nq, Nk, d, layout):
    q, k, v = (t[..., :d] for t in U.make_qkv(B, Hq, Hkv, Nq, Nk, 128, seed=Nk + d, device=DEV, layout=layout))
    v = v * torch.arange(1, Hkv + 1, device=DEV).view((1, -1, 1, 1) if layout == "HND" else (1, 1, -1, 1)).to(v.dtype)
    out = sa.sageattn(q, k, v, tensor_layout=layout, is_causal=True, sm_scale=0.1, check_status=True)
    q, k, v = (torch.nn.functional.pad(t, (0, 128 - d)) for t in (q, k, v))
    want = sa.fp4_attention(sa.quantize_qkv(q, k, v, tensor_layout=layout), is_causal=True, sm_scale=0.1, tensor_layout=layout)
    assert sage3.accuracy(out.float().cpu(), want[..., :d].float().cpu())[1] <= 1e-3


def test_few_query_rows_in_other_layouts():
    q, k, v = U.make_qkv(2, 8, 2, 3, 1300, 128, seed=5, device=DEV)
    want = sa.sageattn(q, k, v, is_causal=True)
    nhd = [t.transpose(1, 2).contiguous() for t in (q, k, v)]
    assert torch.equal(sa.sageattn(*nhd, tensor_layout="NHD", is_causal=True).transpose(1, 2), want)
    narrow = sa.sageattn(q[..., :72], k[..., :72], v[..., :72], sm_scale=0.1)
    full = sa.sageattn(*(torch.nn.functional.pad(t[..., :72], (0, 56)) for t in (q, k, v)), sm_scale=0.1)
    assert torch.equal(narrow, full[..., :72])
    # more queries than keys cannot be few; no key smoothing and one mean per sequence can
    for kw in ({"smooth_k": False}, {"per_block_mean": False}):
        a = sa.sageattn3_blackwell(q, k, v, **kw)
        assert torch.isfinite(a).all() and sage3.accuracy(a.float().cpu(), sa.sageattn(q, k, v).float().cpu())[0] > 0.9


# the workspace that sage3_attention_workspace asks for is enough, and all that is written; one byte less is refused
@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,D,lse", [(2, 8, 2, 1, 1300, 128, True), (1, 8, 1, 8, 3000, 64, False), (1, 4, 2, 300, 500, 128, True)])
def test_workspace_is_not_overrun(B, Hq, Hkv, Nq, Nk, D, lse):
    import ctypes as C
    from sageattention_b200 import _lib
    lib = _lib.load()
    q, k, v = U.make_qkv(B, Hq, Hkv, Nq, Nk, D, seed=Nk, device=DEV)
    want = sa.sageattn(q, k, v, return_lse=True)
    n = C.c_size_t()
    a = _lib.FwdArgs()
    a.shape = _lib.Shape(B, Hq, Hkv, Nq, Nk, D)
    a.per_block_mean = a.smooth_k = 1
    assert lib.sage3_attention_workspace(C.byref(a.shape), 1, C.byref(n)) == _lib.OK
    ws = torch.full((n.value + 65536,), 0xA5, dtype=torch.uint8, device=DEV)
    out, lse_out = torch.empty_like(q), torch.empty(B, Hq, Nq, dtype=torch.float32, device=DEV)
    for t, x in (("q", q), ("k", k), ("v", v)):
        setattr(a, t, _lib.Tensor(None, x.stride(0), x.stride(1), x.stride(2)))
    a.out_stride_b, a.out_stride_h, a.out_stride_n = out.stride(0), out.stride(1), out.stride(2)
    stream = torch.cuda.current_stream().cuda_stream
    for nbytes, status in ((n.value - 1, _lib.ERR_ARGUMENT), (n.value, _lib.OK)):
        a.workspace_bytes = nbytes
        assert lib.sage3_attention_run(C.byref(a), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                                       lse_out.data_ptr() if lse else None, ws.data_ptr(), None, stream) == status
    torch.cuda.synchronize()
    assert bool((ws[n.value:] == 0xA5).all())
    if lse:
        assert torch.equal(out, want[0]) and torch.equal(lse_out, want[1])
    else:
        assert torch.equal(out, sa.sageattn(q, k, v))
