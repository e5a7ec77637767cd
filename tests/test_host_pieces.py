"""``sageattn_from_host``: how host tensors are cut into pieces, what is refused before the device is touched (CPU), and pieces
of every kind through the GPU."""
import pytest
import torch

import sageattention_b200 as sa
from sageattention_b200 import api
from tests import _util as U

MB = 1 << 20


# small entries, several to a piece; entries cut into heads with and without room for the ramp; one head; fewer pieces asked for
# than the size would give; lists
@pytest.mark.parametrize("B,Hkv,head_bytes,head_chunks,want", [
    (5, 4, MB, 8, [(0, 3, 0, 4), (3, 5, 0, 4)]),
    (2, 4, 40 * MB, 1, [(0, 1, 0, 4), (1, 2, 0, 4)]),
    (1, 1, 500 * MB, 8, [(0, 1, 0, 1)]),
    (2, 8, 6 * MB, 8, [(0, 1, 0, 1), (0, 1, 1, 3), (0, 1, 3, 7), (0, 1, 7, 8), (1, 2, 0, 4), (1, 2, 4, 5), (1, 2, 5, 7), (1, 2, 7, 8)]),
    (1, 3, 8 * MB, 8, None), (3, 7, 9 * MB, 2, None), (1, 40, 25 * MB, 8, None), (1, 40, 25 * MB, 16, None), (4, 32, 3 * MB, 5, None),
    (2, 4, MB, [1, 3], [(0, 1, 0, 1), (0, 1, 1, 4), (1, 2, 0, 1), (1, 2, 1, 4)])])
def test_pieces_cover_every_head_once(B, Hkv, head_bytes, head_chunks, want):
    pieces = api._host_pieces(B, Hkv, head_bytes, head_chunks)
    if want is not None:
        assert pieces == want
    heads = [(b, h) for b0, b1, h0, h1 in pieces for b in range(b0, b1) for h in range(h0, h1)]
    assert heads == [(b, h) for b in range(B) for h in range(Hkv)]
    assert all(h1 - h0 == Hkv or b1 - b0 == 1 for b0, b1, h0, h1 in pieces)          # contiguous in [B, H, N, D]
    if isinstance(head_chunks, int):
        # beside the ramp of at most 1 + 2 + 4 heads at either end, at most that many pieces per entry
        most = max(h1 - h0 for _, _, h0, h1 in pieces)
        assert most >= -(-Hkv // head_chunks) or B * Hkv < 16
        assert len(pieces) <= B * head_chunks + 8


def test_bad_piece_lists_are_refused():
    for bad in ([1, 2], [4, 0], [5, -1]):
        with pytest.raises(ValueError):
            api._host_pieces(1, 4, MB, bad)


def test_bad_arguments_are_refused_before_the_device_is_touched(monkeypatch):
    def touched(*a, **k):
        raise RuntimeError("device touched")
    monkeypatch.setattr(torch.cuda, "current_device", touched)
    monkeypatch.setattr(torch.cuda, "current_stream", touched)
    t = lambda *s, dtype=torch.bfloat16: torch.zeros(s, dtype=dtype)
    q, k = t(1, 4, 64, 64), t(1, 2, 64, 64)
    for args, kw, err in [((q.float(), k, k), {}, AssertionError), ((q, k, k.half()), {}, AssertionError),
                          ((t(1, 3, 64, 64), k, k), {}, ValueError), ((q, k, t(1, 2, 65, 64)), {}, ValueError),
                          ((q, t(1, 2, 64, 32), t(1, 2, 64, 32)), {}, ValueError), ((t(4, 64, 64), k, k), {}, ValueError),
                          ((t(1, 2, 8, 136), t(1, 2, 8, 136), t(1, 2, 8, 136)), {}, ValueError),
                          ((q, k, k), {"attn_mask": k}, NotImplementedError), ((q, k, k), {"return_lse": True}, TypeError),
                          ((q, k, k), {"head_chunks": [3]}, ValueError)]:
        with pytest.raises(err):
            sa.sageattn_from_host(*args, **kw)
    with pytest.raises(RuntimeError, match="device touched"):
        sa.sageattn_from_host(q, k, k)


@pytest.mark.gpu
@pytest.mark.parametrize("B,Hq,Hkv,head_chunks,n", [(2, 16, 8, 8, 8), (1, 14, 14, 3, 6), (3, 4, 4, 8, 12), (2, 8, 4, [3, 1], 4), (1, 6, 3, 1, 1)])
def test_head_pieces_match_the_device_operator(monkeypatch, B, Hq, Hkv, head_chunks, n):
    """The sizes that go in pieces of heads take gigabytes; the same cuts are made here by a smaller piece."""
    q, k, v = U.make_qkv(B, Hq, Hkv, 200, 300, 64, seed=B + Hq)
    head = (q.numel() + k.numel() + v.numel()) * 2 // (B * Hkv)
    monkeypatch.setattr(api, "_host_piece_bytes", lambda total: min(4, Hkv - 1) * head if Hkv > 4 else head)
    assert len(api._host_pieces(B, Hkv, head, head_chunks)) == n
    want = sa.sageattn(q.cuda(), k.cuda(), v.cuda(), is_causal=True).cpu()
    for _ in range(2):
        got = sa.sageattn_from_host(q.pin_memory(), k.pin_memory(), v.pin_memory(), head_chunks=head_chunks, is_causal=True)
        torch.cuda.synchronize()
        assert torch.equal(got, want)


@pytest.mark.gpu
def test_a_failing_piece_leaves_nothing_under_way(monkeypatch):
    """The buffers go back to the current stream's pool: that stream has to wait for the copies into them, also when a
    piece fails behind them."""
    q, k, v = (t.pin_memory() for t in U.make_qkv(1, 4, 4, 300, 300, 128, seed=3))
    want = sa.sageattn_from_host(q, k, v)                        # (makes the streams)
    torch.cuda.synchronize()
    s_in = api._host_streams[torch.device("cuda", torch.cuda.current_device())][0]

    def fail(*a, **kw):
        with torch.cuda.stream(s_in):
            torch.cuda._sleep(int(2e8))                          # what is queued behind the copies: about 0.1 s
        raise KeyError("piece")
    with monkeypatch.context() as m:
        m.setattr(api, "sageattn3_blackwell", fail)
        with pytest.raises(KeyError):
            sa.sageattn_from_host(q, k, v, head_chunks=[1, 3])
    assert not s_in.query()
    torch.cuda.current_stream().synchronize()
    assert s_in.query()
    got = sa.sageattn_from_host(q, k, v)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
