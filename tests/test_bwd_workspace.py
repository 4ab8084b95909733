"""CPU: scratch of the chunked backward, by the kernels that a call takes."""
import ctypes

import pytest

from nha_b200 import _lib


def _bytes(N, Ttot, HQ, H, K, M, scale=0.125):
    d = _lib.ChunkDesc()
    d.N, d.Ttot, d.HQ, d.H, d.K, d.V, d.M, d.scale = N, Ttot, HQ, H, K, K, M, scale
    return _lib.load().nha_chunk_bwd_workspace_bytes(ctypes.byref(d))


@pytest.mark.parametrize('N,T,HQ,H,M', [(16, 2048, 16, 16, 64), (3, 999, 8, 2, 32), (1, 1, 1, 1, 8)])
def test_head_dim_64_lays_out_what_its_kernels_use(N, T, HQ, H, M, monkeypatch):
    monkeypatch.delenv('NHA_B200_NO_UMMA', raising=False)
    tokens, chunks = N * T, _lib.load().nha_chunk_count_bound(N * T, N)
    # delta and the joint log-sum-exp; the slot part of dv and ds of steep chunks; the states' gradients and the chunks' decays: fp32
    used = 4 * (2 * tokens * HQ + tokens * H * (64 + M) + chunks * H * (2 * 64 * M + M))
    got = _bytes(N, tokens, HQ, H, 64, M)
    assert used <= got <= used + 7 * 256
    # the general kernels need more, also where only the scale keeps the others from running
    assert _bytes(N, tokens, HQ, H, 64, M, scale=-0.125) > got
    monkeypatch.setenv('NHA_B200_NO_UMMA', '1')
    assert _bytes(N, tokens, HQ, H, 64, M) == _bytes(N, tokens, HQ, H, 64, M, scale=-0.125) > got
