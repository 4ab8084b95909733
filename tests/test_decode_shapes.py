"""CPU: the operators refuse, on the host and before anything is launched, tensors that do not hold what the kernel would
read through their pointers.  The tensors are host tensors: right shapes get as far as the device check behind the shape checks."""
import pytest
import torch

import nha_b200

B, HQ, H, K, V, M, W = 3, 4, 2, 32, 48, 16, 8
BAD = {                                          # one axis of one tensor at a time
    'k': [(1, 1, H, K), (B, 2, H, K), (B, 1, 1, K), (B, 1, H, K // 2)], 'v': [(1, 1, H, V), (B, 2, H, V), (B, 1, 1, V)],
    'g': [(1, 1, H, M), (B, 2, H, M), (B, 1, 1, M)], 's': [(1, 1, H, M), (B, 1, H, M // 2)], 'q': [(1, 1, HQ, K), (B, 1, 3, K), (B, 1, HQ, K // 2)],
    'sw_k': [(1, W, H, K), (B, W - 1, H, K), (B, W, H, K // 2)], 'sw_v': [(1, W, H, V), (B, W - 1, H, V), (B, W, 1, V), (B, W, H, V // 2)],
    'cos': [(1, W - 1, K), (2, W, K), (1, W, K // 2)], 'hk': [(1, H, K, M), (B, H, K, M // 2)], 'hv': [(1, H, M, V), (B, H, M // 2, V)],
}
SHAPES = dict(q=(B, 1, HQ, K), k=(B, 1, H, K), v=(B, 1, H, V), g=(B, 1, H, M), s=(B, 1, H, M), sw_k=(B, W, H, K), sw_v=(B, W, H, V),
              cos=(1, W, K), hk=(B, H, K, M), hv=(B, H, M, V))


def _call(op, **changed):
    x = {n: torch.zeros(s) if n in ('hk', 'hv') else torch.zeros(s, dtype=torch.bfloat16) for n, s in {**SHAPES, **changed}.items()}
    x['sin'] = x['cos']
    x['initial_state'] = (x.pop('hk'), x.pop('hv'))
    return op(**x, output_final_state=True)


@pytest.mark.parametrize('op', [nha_b200.fused_recurrent_nha_decode, nha_b200.fused_recurrent_nha_decode_bf16_state])
def test_decode(op):
    with pytest.raises(AssertionError, match='CUDA library only'):
        _call(op)
    for name, shapes in BAD.items():
        for shape in shapes:
            with pytest.raises(AssertionError) as e:
                _call(op, **{name: shape})
            assert 'CUDA' not in str(e.value), (name, shape, str(e.value))


@pytest.mark.parametrize('layout', ['fused', 'two launches', 'rotated'])
def test_decode_ring(layout):
    from nha_b200.ring_cache import RingLayer, fused_recurrent_nha_decode_ring
    D = K

    def call(layer_change=lambda y: None, cos=(1, W, D), **changed):
        y = RingLayer(*(torch.zeros(B, W, H, n) for n in (D, D, M)), torch.zeros(B, H, D, M), torch.zeros(B, H, M, D), fused=layout == 'fused')
        if layout == 'rotated':
            y.ring_kr = torch.zeros_like(y.ring_k)
        layer_change(y)
        x = {**dict(q=(B, 1, HQ, D), k=(B, 1, H, D), v=(B, 1, H, D), g=(B, 1, H, M)), **changed}
        x = {n: torch.zeros(s, dtype=torch.bfloat16) for n, s in x.items()}
        head, rings = y.head.clone(), [r.clone() for r in (y.ring_k, y.ring_v, y.ring_g)]
        try:
            fused_recurrent_nha_decode_ring(**x, layer=y, cos=torch.zeros(cos), sin=torch.zeros(cos))
        finally:
            assert y.fill == W and torch.equal(y.head[:, :1] if y.head.dim() > 1 else y.head, head[:, :1] if head.dim() > 1 else head)
            assert all(torch.equal(a, b) for a, b in zip((y.ring_k, y.ring_v, y.ring_g), rings))

    def cut(name, *index):
        return lambda y: setattr(y, name, getattr(y, name)[index].contiguous())

    bad = [dict(k=(1, 1, H, D)), dict(k=(B, 1, H, D // 2)), dict(v=(1, 1, H, D)), dict(v=(B, 2, H, D)), dict(g=(1, 1, H, M)), dict(g=(B, 1, H, M // 2)),
           dict(q=(1, 1, HQ, D)), dict(cos=(2, W, D)), dict(cos=(1, W, D // 2)),
           *(dict(layer_change=cut(n, slice(1))) for n in ('ring_k', 'ring_v', 'ring_g', 'hk', 'hv', 'head')),
           dict(layer_change=lambda y: setattr(y, 'hk', y.hk.bfloat16())), dict(layer_change=lambda y: setattr(y, 'ring_k', y.ring_k.float())),
           dict(layer_change=lambda y: setattr(y, 'ring_v', y.ring_v.transpose(2, 3)))]
    for change in bad:
        with pytest.raises(AssertionError) as e:
            call(**change)
        assert 'CUDA' not in str(e.value), (change, str(e.value))


def test_recurrent():
    def call(**changed):
        x = {**dict(q=(B, 1, HQ, K), k=(B, 1, H, K), v=(B, 1, H, V), sliding_window=(B, 1, HQ, W), s=(B, 1, H, M), g=(B, 1, H, M)), **changed}
        nha_b200.fused_recurrent_nha(**{n: torch.zeros(s, dtype=torch.bfloat16) for n, s in x.items()})

    with pytest.raises(AssertionError, match='CUDA library only'):
        call()
    for change in (dict(k=(1, 1, H, K)), dict(k=(B, 1, H, K // 2)), dict(v=(1, 1, H, V)), dict(s=(B, 1, H, M // 2)), dict(g=(1, 1, H, M)),
                   dict(sliding_window=(1, 1, HQ, W)), dict(q=(1, 1, HQ, K))):
        with pytest.raises(AssertionError) as e:
            call(**change)
        assert 'CUDA' not in str(e.value), (change, str(e.value))


def test_chunk_operators_take_tensors_of_the_gpu():
    T = 5
    x = {n: torch.zeros(B, T, HQ if n[0] == 'q' else H, {'s': M, 'g': M, 'v': V}.get(n, K), dtype=torch.bfloat16)
         for n in ('q_swa', 'k_swa', 'q_gsa', 'k_gsa', 'v', 's', 'g')}
    with pytest.raises(AssertionError, match='CUDA library only'):
        nha_b200.chunk_nha(**x, window_size_left=4, window_size_right=0)
    with pytest.raises(AssertionError, match='CUDA library only'):
        nha_b200.fused_chunk_nha_prefill(x['q_gsa'], x['k_gsa'], x['v'], x['q_swa'], x['k_swa'], x['s'], x['g'], 4)


@pytest.mark.parametrize('want,B,H,D,W,splits', [
    # us a layer without and with the prefetch differ by more than 2 % at each of these (64 slots, fp32 state)
    (True, 24, 4, 128, 512, 2), (True, 12, 4, 128, 1200, 4), (True, 64, 4, 128, 128, 1), (True, 112, 4, 128, 128, 1), (True, 80, 16, 64, 128, 1),
    (False, 36, 4, 128, 512, 2), (False, 40, 4, 128, 512, 1), (False, 48, 4, 128, 512, 1), (False, 56, 4, 128, 512, 1), (False, 20, 8, 128, 512, 1),
    (False, 28, 8, 128, 512, 1), (False, 16, 4, 128, 1200, 4), (False, 24, 4, 128, 1200, 2)])
def test_the_window_is_prefetched_where_that_measured_faster(want, B, H, D, W, splits):
    import ctypes
    from nha_b200 import _lib
    rule = _lib.load()['_ZN3nha19decode_window_aheadEiiiiiiiiil']         # nha::decode_window_ahead, not part of the C ABI
    rule.restype, rule.argtypes = ctypes.c_bool, [ctypes.c_int] * 9 + [ctypes.c_int64]
    assert rule(B, H, D, 64, W, splits, 4, 2, 148, 132644864) is want
