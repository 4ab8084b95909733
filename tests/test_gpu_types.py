"""GPU: the operators on fp32 and fp16 tensors.  Inputs are rounded to bf16 on the way in and results converted on the way out, so a
call must give the bits of the bf16 call; the conversion kernel is also checked by itself, at sizes that end inside its pieces of eight,
with pointers off its 16 bytes, and on values where rounding shows."""
import ctypes

import pytest
import torch

from tests import inputs as gen
from tests.test_gpu_decode import _off_16

pytestmark = pytest.mark.gpu
NAMES = ('q_swa', 'k_swa', 'q_gsa', 'k_gsa', 'v', 's', 'g')
WIDE = [torch.float32, torch.float16]


def _wider(t, dt):
    """Values that bf16 does not hold."""
    return t.cuda().to(dt) * (1 + 2.0 ** -9)


@pytest.mark.parametrize('dt', WIDE)
@pytest.mark.parametrize('D,T,off', [(64, 130, False), (128, 77, True)])
def test_chunk(dt, D, T, off):
    from nha_b200 import chunk_nha
    d = gen.layer_inputs(21, 1, T, 2, 2, D, D, 64)
    wide = [_wider(d[n], dt) for n in NAMES]
    do = _wider(d['do'], dt)
    how = dict(window_size_left=64, window_size_right=0, output_final_state=True)
    x = [(_off_16(t) if off else t).detach().requires_grad_(True) for t in wide]
    b = [t.bfloat16().requires_grad_(True) for t in wide]
    got, want = chunk_nha(*x, **how), chunk_nha(*b, **how)
    assert got[0].dtype == dt and torch.equal(got[0], want[0].to(dt))
    for i in (1, 2):
        assert torch.equal(got[i], want[i])
    assert torch.equal(got[3][0], want[3][0]) and torch.equal(got[3][1], want[3][1])
    for a, c in zip(torch.autograd.grad(got[0], x, do), torch.autograd.grad(want[0], b, do.bfloat16())):
        assert a.dtype == dt and torch.equal(a, c.to(dt))


@pytest.mark.parametrize('dt', WIDE)
def test_prefill_and_decode(dt):
    from nha_b200 import fused_chunk_nha_prefill, fused_recurrent_nha, fused_recurrent_nha_decode
    d = gen.prefill_inputs(22, 2, 2, 2, 64, 64, 64, 64, 100, False)
    names = ('q', 'k', 'v', 'rotary_q', 'rotary_k', 's', 'g')
    wide = [_wider(d[n], dt) for n in names]
    o, (hk, hv) = fused_chunk_nha_prefill(*wide, 64, output_final_state=True)
    ob, (hkb, hvb) = fused_chunk_nha_prefill(*(t.bfloat16() for t in wide), 64, output_final_state=True)
    assert o.dtype == dt and torch.equal(o, ob.to(dt)) and torch.equal(hk, hkb) and torch.equal(hv, hvb)
    c = gen.decode_inputs(23, 2, 2, 2, 64, 64, 64, 64)
    names = ('q', 'k', 'v', 'g', 'sw_k_raw', 'vw', 'cos', 'sin')
    wide = {n: _wider(c[n], dt) for n in names}
    run = lambda y: fused_recurrent_nha_decode(*(y[n] for n in names[:6]), cos=y['cos'], sin=y['sin'],  # noqa: E731
                                               initial_state=(c['hk0'].cuda(), c['hv0'].cuda()), output_final_state=True)
    (o, s), (ob, sb) = run(wide), run({n: t.bfloat16() for n, t in wide.items()})
    assert o.dtype == dt and torch.equal(o, ob.to(dt)) and torch.equal(s[0], sb[0]) and torch.equal(s[1], sb[1])
    names = ('q', 'k', 'v', 'sliding_window', 's', 'g')
    wide = [_wider(c[n], dt) for n in names]
    o, p, _ = fused_recurrent_nha(*wide)
    ob, pb, _ = fused_recurrent_nha(*(t.bfloat16() for t in wide))
    assert o.dtype == dt and torch.equal(o, ob.to(dt)) and torch.equal(p, pb)


@pytest.mark.parametrize('dt', WIDE)
@pytest.mark.parametrize('back', [False, True])
@pytest.mark.parametrize('off', [False, True])
def test_the_conversion_kernel(dt, back, off):
    from nha_b200 import _lib
    src, dst = (torch.bfloat16, dt) if back else (dt, torch.bfloat16)
    code = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}                 # NHA_BF16, NHA_FP16, NHA_FP32
    special = torch.tensor([0.0, -0.0, 1 + 2.0 ** -8, 1 + 3 * 2.0 ** -8, 1 + 2.0 ** -8 + 2.0 ** -10, 2.0 ** -14, 65504.0, -65504.0, float('inf'), float('-inf'), float('nan')])
    xs = [torch.randn(n, generator=torch.Generator().manual_seed(n)).cuda() for n in (1, 7, 8, 9, 2055, 300001, 16)] + [special.cuda()]
    xs = [x.to(src) for x in xs]
    ys = [torch.full_like(x, 7.0, dtype=dst) for x in xs]
    if off:
        xs, ys = [_off_16(x) for x in xs], [_off_16(y) for y in ys]
    n = len(xs)
    ptrs = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() for t in ts])  # noqa: E731
    st = _lib.load().nha_cast_many(ptrs(xs), ptrs(ys), (ctypes.c_int64 * n)(*[t.numel() for t in xs]), n, code[src], code[dst],
                                   torch.cuda.current_stream().cuda_stream)
    assert st == 0
    for x, y in zip(xs, ys):
        assert torch.equal(torch.nan_to_num(x.to(dst), nan=5.0), torch.nan_to_num(y, nan=5.0)) and torch.equal(torch.isnan(x), torch.isnan(y))
