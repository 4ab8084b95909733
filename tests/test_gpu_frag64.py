"""GPU: the head-dim-64 kernels with full lanes: every slot count they take, ragged last chunks, windows of one and of several
steps, window logits that grow towards older keys (the running reference of the softmax is raised), against the oracle."""
import pytest
import torch

from oracle import nha_oracle as orc
from tests import inputs as gen
from tests.gpu_util import TOL_OUT, assert_close
from tests.test_gpu_chunk import compare, run_gpu, run_oracle

pytestmark = pytest.mark.gpu
NAMES = ('q_swa', 'k_swa', 'q_gsa', 'k_gsa', 'v', 's', 'g')


@pytest.mark.parametrize('M', [16, 32, 48, 64])
@pytest.mark.parametrize('HQ,H,T,wl,shift', [(2, 2, 129, 64, 0), (6, 2, 65, 63, 64), (2, 1, 400, 300, 0), (1, 1, 700, -1, 70)])
def test_forward(M, HQ, H, T, wl, shift):
    from nha_b200 import chunk_nha
    d = gen.layer_inputs(50 + M + T, 1, T, HQ, H, 64, 64, M, gate_div=2.0, val_scale=1.0)
    grow = torch.linspace(6.0, 0.2, T)[None, :, None, None]
    d['k_swa'] = (d['k_swa'].float() * grow).bfloat16()            # older keys have the larger logits
    want = orc.nha_varlen(*(d[n][0].double() for n in ('q_gsa', 'q_swa', 'k_gsa', 'k_swa', 'v', 's', 'g')), [0, T], 0.125, wl, shift, None, None)
    got = chunk_nha(*(d[n].cuda() for n in NAMES), window_size_left=wl, window_size_right=0, gsa_kv_shift=shift, output_final_state=True)
    for x, y, name in zip((got[0][0], got[1][0], got[2][0], *got[3]), want, ('o', 'lse_swa', 'lse_gsa', 'hk', 'hv')):
        assert_close(x, y, TOL_OUT, name)


@pytest.mark.parametrize('M', [16, 32, 48, 64])
@pytest.mark.parametrize('HQ,H,cu,wl,shift', [(2, 2, [0, 64, 193], 64, 0), (3, 1, [0, 1, 130], [0, 63], 64), (4, 2, [0, 321], 200, 65),
                                              (1, 1, [0, 257], -1, 0)])
def test_backward(M, HQ, H, cu, wl, shift, D=64):
    T = cu[-1]
    d = {n: x[0] for n, x in gen.layer_inputs(70 + M + T, 1, T, HQ, H, D, D, M, gate_div=2.0, val_scale=1.0).items() if torch.is_tensor(x)}
    ge = torch.Generator().manual_seed(M + T)
    do, dlse = torch.randn(T, HQ, D, generator=ge).bfloat16(), 0.1 * torch.randn(T, HQ, generator=ge)
    N = len(cu) - 1
    dhk, dhv = 0.1 * torch.randn(N, H, D, M, generator=ge), 0.1 * torch.randn(N, H, M, D, generator=ge)
    wls = wl if isinstance(wl, list) else [wl] * N
    want, gwant = run_oracle(d, cu, D ** -0.5, wls, [shift] * N, None, None, do, dlse, dhk, dhv)
    got, ggot = run_gpu(d, cu, max(b - a for a, b in zip(cu, cu[1:])), D ** -0.5, wls, [shift] * N, None, None, do, dlse, dhk, dhv)
    compare(got, ggot, want, gwant)


@pytest.mark.parametrize('HQ,H,cu,wl,shift', [(2, 2, [0, 64, 193], 64, 0), (4, 1, [0, 1, 130], [0, 63], 64), (4, 2, [0, 321], 200, 65),
                                              (2, 1, [0, 257], -1, 0), (3, 1, [0, 191], 127, 128)])
def test_backward_128(HQ, H, cu, wl, shift):
    test_backward(64, HQ, H, cu, wl, shift, D=128)


def test_backward_128_repeatable():
    # many chunks in flight, several window tiles, several heads a group: tiles that were read before they arrived would show as
    # differences between two runs
    from nha_b200 import chunk_nha
    d = gen.layer_inputs(91, 2, 1999, 16, 4, 128, 128, 64)
    do = d['do'].cuda()
    runs = []
    for _ in range(4):
        x = [d[n].cuda().requires_grad_(True) for n in NAMES]
        o = chunk_nha(*x, window_size_left=200, window_size_right=0, gsa_kv_shift=128)[0]
        runs.append(torch.autograd.grad(o, x, do))
    for other in runs[1:]:
        for a, b, n in zip(runs[0], other, NAMES):
            assert torch.equal(a, b), n


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('wl', [20, 150])
@pytest.mark.parametrize('which', ['q_swa', 'k_swa'])
def test_a_nan_in_the_window_shows_in_every_row_that_sees_it(D, wl, which):
    from nha_b200 import chunk_nha
    T, at = 330, 70
    d = gen.layer_inputs(92, 1, T, 2, 2, D, D, 64)
    run = lambda: chunk_nha(*(d[n].cuda() for n in NAMES), window_size_left=wl, window_size_right=0)[:2]  # noqa: E731
    o0, lse0 = run()
    d[which][0, at, 1, 3] = float('nan')
    o, lse = run()
    sees = torch.zeros(T, dtype=torch.bool, device='cuda')
    sees[at:at + (wl + 1 if which == 'k_swa' else 1)] = True
    assert torch.isnan(o[0, sees, 1]).all() and torch.isnan(lse[0, sees, 1]).all()
    assert torch.equal(o[0, ~sees], o0[0, ~sees]) and torch.equal(o[0, :, 0], o0[0, :, 0]) and torch.equal(lse[0, ~sees], lse0[0, ~sees])


def test_a_single_window_key_gives_its_logit_exactly():
    # whole numbers: the product is exact, the scale 1/8 too, and the log-sum-exp over one key is its logit
    from nha_b200 import chunk_nha
    d = gen.layer_inputs(93, 1, 200, 2, 2, 64, 64, 64)
    q, k = (torch.randint(-8, 9, d[n].shape, generator=torch.Generator().manual_seed(i)) for i, n in enumerate(('q_swa', 'k_swa')))
    d['q_swa'], d['k_swa'] = q.bfloat16(), k.bfloat16()
    lse = chunk_nha(*(d[n].cuda() for n in NAMES), window_size_left=0, window_size_right=0)[1]
    assert torch.equal(lse.cpu(), (q * k).sum(-1).float() / 8)


@pytest.mark.parametrize('M', [32, 64])
@pytest.mark.parametrize('D,wl,shift', [(64, 64, 0), (64, 63, 64), (128, 127, 128)])
def test_gradients_at_the_gates_of_training(M, D, wl, shift):
    # gate logits ~ N(0, 1) undivided.  The gradient of the gates is a difference of large terms: 1.9e-2 to 2.1e-2 from 64 bits on the
    # tensor-core and on the general kernels alike (16 inputs each); the others stay below 6e-3
    from nha_b200 import chunk_nha
    d = gen.layer_inputs(94 + M, 1, 300, 4, 4, D, D, M, gate_div=1.0)
    xs = [d[n].double()[0].requires_grad_(True) for n in NAMES]
    y = dict(zip(NAMES, xs))
    o = orc.nha_sequence(y['q_gsa'], y['q_swa'], y['k_gsa'], y['k_swa'], y['v'], y['s'], y['g'], D ** -0.5, wl, shift)[0]
    want = torch.autograd.grad(o, xs, d['do'].double()[0])
    x = [d[n].cuda().requires_grad_(True) for n in NAMES]
    got = torch.autograd.grad(chunk_nha(*x, window_size_left=wl, window_size_right=0, gsa_kv_shift=shift)[0], x, d['do'].cuda())
    for n, a, b in zip(NAMES, got, want):
        assert_close(a[0], b, 2.6e-2 if n == 'g' else 8e-3, n)
