"""GPU: the slot branch's backward walk at head dim 64, where it can go wrong.

A run of chunks starts either at the end of a sequence or from the scan over the terms of the chunks behind it.  Which of the two, and how
long the runs are, depends on how the same sequences are handed in; the gradients must not, to the bit.
"""
import pytest
import torch

from tests import inputs as gen
from tests.gpu_util import TOL_GRAD, assert_close
from tests.test_gpu_chunk import NAMES, flat_inputs, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


def _grads(x, do, B, T, how, **kw):
    from nha_b200 import chunk_nha
    leaves = {n: (x[n][None] if how == 'packed' else x[n].view(B, T, *x[n].shape[1:])).detach().cuda().requires_grad_(True) for n in NAMES}
    if how == 'packed':
        kw.update(cu_seqlens=torch.arange(0, (B + 1) * T, T, dtype=torch.int32, device='cuda'), max_seqlen=B * T)
    o, _, lse = chunk_nha(*(leaves[n] for n in ('q_swa', 'k_swa', 'q_gsa', 'k_gsa', 'v', 's', 'g')), window_size_right=0, **kw)
    loss = (o.reshape(do.shape).float() * do.cuda()).sum() + 0.1 * lse.sum()
    return dict(zip(NAMES, torch.autograd.grad(loss, [leaves[n] for n in NAMES])))


# 320 sequences give every kv head whole sequences to walk; packed, with a bound on the lengths that does not say so, the same calls take the terms,
# the scan and runs that cut sequences
@pytest.mark.parametrize('T', [1, 63, 64, 65, 200, 449])
def test_whole_sequences_and_runs_from_the_scan_agree_to_the_bit(T):
    B, H, M = 80, 4, 64
    d = gen.layer_inputs(31 + T, B, T, H, H, 64, 64, M, gate_div=1.0)
    x, do = flat_inputs(d, B, T), d['do'].reshape(B * T, H, 64).float()
    a = _grads(x, do, B, T, 'dense', window_size_left=64, gsa_kv_shift=0)
    b = _grads(x, do, B, T, 'packed', window_size_left=64, gsa_kv_shift=0)
    for n in NAMES:
        assert torch.equal(a[n].reshape(-1), b[n].reshape(-1)), n


# Packed sequences that the true longest length sends down the walk over whole sequences, and a looser bound through the scan: unequal lengths, empty
# sequences (first, last and between), the states' gradients
@pytest.mark.parametrize('HQ,H', [(4, 4), (8, 4)])
def test_packed_whole_sequences_and_runs_agree_to_the_bit(HQ, H):
    lens = [0, 65, 1, 0, 64, 200, 63, 0, 130, 128, 0] + [40 + 7 * i for i in range(20)] + [0]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    N, T, M = len(lens), cu[-1], 64
    d = gen.layer_inputs(77, 1, T, HQ, H, 64, 64, M, gate_div=1.0)
    x, do = flat_inputs(d, 1, T), d['do'].reshape(T, HQ, 64).float()
    torch.manual_seed(5)
    state = (torch.randn(N, H, 64, M) * 0.5, torch.randn(N, H, M, 64) * 0.5)
    end = (torch.randn(N, H, 64, M) * 0.1, torch.randn(N, H, M, 64) * 0.1)
    _, a = run_gpu(x, cu, max(lens), 0.125, 64, 0, *state, do, None, *end)
    _, b = run_gpu(x, cu, T, 0.125, 64, 0, *state, do, None, *end)
    for n in a:
        assert torch.equal(a[n], b[n]), n
    empty = [i for i, n in enumerate(lens) if n == 0]
    assert torch.equal(a['hk0'][empty].cpu().float(), end[0][empty]) and torch.equal(a['hv0'][empty].cpu().float(), end[1][empty])


# one and several heads a kv head, fewer than 64 slots, ragged ends, a shift that is not a whole chunk, with and without a gradient on lse_gsa,
# and chunks too steep for one decay reference in the middle of a run and at its end
@pytest.mark.parametrize('HQ,H,M,T,shift,steep,dlse', [(2, 2, 64, 641, 0, False, False), (2, 2, 64, 640, 33, True, True), (1, 1, 16, 200, 65, False, True),
                                                       (6, 2, 64, 321, 0, True, False), (4, 1, 48, 257, 128, False, True), (1, 1, 32, 130, 0, True, True)])
def test_walk_against_the_oracle(HQ, H, M, T, shift, steep, dlse):
    d = gen.layer_inputs(500 + T, 1, T, HQ, H, 64, 64, M, gate_div=1.0, val_scale=1.0)
    if steep:
        g = d['g'].float()
        g[:, 20:60] = g[:, 20:60] * 3 - 1
        g[:, -70:] = g[:, -70:] * 3 - 1
        d['g'] = g.to(torch.bfloat16)
        d['s'] = (1 - d['g'].float().exp()).to(torch.bfloat16)
    x, do = flat_inputs(d, 1, T), d['do'].reshape(T, HQ, 64).float()
    torch.manual_seed(T)
    dl = torch.randn(T, HQ) * 0.1 if dlse else None
    state = (torch.randn(1, H, 64, M) * 0.5, torch.randn(1, H, M, 64) * 0.5)
    end = (torch.randn(1, H, 64, M) * 0.1, torch.randn(1, H, M, 64) * 0.1)
    _, want = run_oracle(x, [0, T], 0.125, 64, shift, *state, do, dl, *end)
    for batched in (1, None):
        _, got = run_gpu(x, [0, T], T, 0.125, 64, shift, *state, do, dl, *end, batched_B=batched)
        for n in want:
            assert torch.isfinite(got[n].float()).all(), n
            assert_close(got[n], want[n], TOL_GRAD, n)


def test_gate_gradients_are_as_precise_as_the_others():
    """p dp and s' ds' of a pair of rows cancel when both are formed from the operands that the products had: the error of dg is that of one
    bf16 rounding (2^-9 each of a few operands, 4e-3 measured) and not that of the difference of two large sums (2e-2)."""
    B, T, H, M = 2, 512, 4, 64
    d = gen.layer_inputs(9, B, T, H, H, 64, 64, M, gate_div=1.0)
    x, do = flat_inputs(d, B, T), d['do'].reshape(B * T, H, 64).float()
    _, want = run_oracle(x, [0, T, 2 * T], 0.125, 64, 0, None, None, do, None)
    _, got = run_gpu(x, [0, T, 2 * T], T, 0.125, 64, 0, None, None, do, None, batched_B=B)
    assert_close(got['g'], want['g'], 4 * 2.0 ** -9, 'g')


# Several query heads a kv head walk whole sequences where those fill the SMs (a CTA an SM, and two), runs from the scan elsewhere
@pytest.mark.parametrize('B,HQ,H,T', [(37, 8, 4, 130), (74, 8, 4, 257), (74, 28, 4, 65)])
def test_grouped_whole_sequences_and_runs_agree_to_the_bit(B, HQ, H, T):
    d = gen.layer_inputs(67 + T, B, T, HQ, H, 64, 64, 64, gate_div=1.0)
    x, do = flat_inputs(d, B, T), d['do'].reshape(B * T, HQ, 64).float()
    a = _grads(x, do, B, T, 'dense', window_size_left=64, gsa_kv_shift=0)
    b = _grads(x, do, B, T, 'packed', window_size_left=64, gsa_kv_shift=0)
    for n in NAMES:
        assert torch.equal(a[n].reshape(-1), b[n].reshape(-1)), n
