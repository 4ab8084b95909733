"""GPU: chunks that decay by more than one reference can carry, inside the backward walk at head dim 64: between others, first, last, several in a row,
in runs of several chunks that start at a sequence's end and in runs that start from the scan."""
import pytest
import torch

from tests import inputs as gen
from tests.gpu_util import TOL_GRAD, assert_close, err
from tests.test_gpu_chunk import NAMES, flat_inputs, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


def _inputs(lens, HQ, H, M, slots):
    T = sum(lens)
    d = gen.layer_inputs(910 + T + HQ, 1, T, HQ, H, 64, 64, M, gate_div=1.0, val_scale=1.0)
    g, at = d['g'].float(), 0
    for n, size in enumerate(lens):
        for c in range((size + 63) // 64):
            last = 64 * c + 64 >= size
            if n % 5 == 4 or (n % 5 == 1 and c == 0) or (n % 5 == 2 and c == 1) or (n % 5 == 3 and last):
                rows = slice(at + 64 * c, at + min(size, 64 * c + 64))
                g[:, rows, :, :slots] = g[:, rows, :, :slots] * 2 - 2.5
        at += size
    d['g'] = g.to(torch.bfloat16)
    d['s'] = (1 - d['g'].float().exp()).to(torch.bfloat16)
    d['g'][:, 70, :, 1] = -200.0                               # one token that forgets a slot at once, beside its weight as it was
    return flat_inputs(d, 1, T), d['do'].reshape(T, HQ, 64).float()


# 80 sequences of 4 kv heads (74, two CTAs an SM, with several query heads): with their longest length every CTA walks whole sequences, with a bound
# that does not say so runs of several chunks that cut them.  All slots of a chunk steep, or a few; a whole number of slots for TMA and fewer; one and two heads a kv head
@pytest.mark.parametrize('HQ,H,M,slots,shift', [(4, 4, 64, 64, 0), (4, 4, 64, 3, 0), (8, 4, 64, 64, 0), (8, 4, 64, 5, 33), (4, 4, 48, 48, 64)])
def test_steep_chunks_inside_runs(HQ, H, M, slots, shift, monkeypatch):
    N = 80 if HQ == H else 74
    lens = [150 + (37 * i) % 151 for i in range(N)]
    x, do = _inputs(lens, HQ, H, M, slots)
    cu = [sum(lens[:i]) for i in range(N + 1)]
    torch.manual_seed(HQ)
    dl = torch.randn(cu[-1], HQ) * 0.1
    state = (torch.randn(N, H, 64, M) * 0.5, torch.randn(N, H, M, 64) * 0.5)
    end = (torch.randn(N, H, 64, M) * 0.1, torch.randn(N, H, M, 64) * 0.1)
    # (both ways form the state gradient by the same arithmetic)
    got, cut = [run_gpu(x, cu, bound, 0.125, 64, shift, *state, do, dl, *end)[1] for bound in (max(lens), cu[-1])]
    for k in got:
        assert torch.isfinite(got[k].float()).all() and torch.equal(got[k], cut[k]), k
    # a few sequences of every kind against the oracle, all rows of a tensor together.  The gate gradients of steep chunks are small differences of
    # large terms: where they leave the bar, no further off than those of the general kernels, which served such chunks before the walk did
    monkeypatch.setenv('NHA_B200_NO_UMMA', '1')
    general = run_gpu(x, cu, max(lens), 0.125, 64, shift, *state, do, dl, *end)[1]
    some, want = (0, 1, 2, 3, 4, N - 1), []
    for n in some:
        a, b = cu[n], cu[n + 1]
        xs = {k: v[a:b] for k, v in x.items()}
        want.append(run_oracle(xs, [0, b - a], 0.125, 64, shift, state[0][n:n + 1], state[1][n:n + 1], do[a:b], dl[a:b], end[0][n:n + 1], end[1][n:n + 1])[1])
    for k in got:
        rows = [slice(n, n + 1) if k in ('hk0', 'hv0') else slice(cu[n], cu[n + 1]) for n in some]
        ref = torch.cat([w[k] for w in want])
        assert_close(torch.cat([got[k][r] for r in rows]), ref, max(TOL_GRAD, err(torch.cat([general[k][r] for r in rows]), ref)), k)
