"""What is measured when the framework is tuned: the calls that a model built on it makes, over the sizes it makes them at.

A case is one of seven kinds of call, each through the public entry points of ``nha_b200``:

``train``      ``chunk_nha`` forward and backward on a batch of equal-length sequences (a training layer)
``packed``     the same on sequences packed with ``cu_seqlens``, a window of its own for each (packed fine-tuning)
``prefill``    ``fused_chunk_nha_prefill`` of a prompt, final slot memory returned (serving, first token)
``decode``     one token for a stack of layers, ``fused_recurrent_nha_decode`` per layer (serving, every other token)
``ring``       the same on ``NHARingCache``, the window update inside the call
``recurrent``  ``fused_recurrent_nha``: one step with window logits that the caller computed
``around``     what the layer runs in front of and behind the operator, forward and backward
"""
import math
import random

import torch
import torch.nn.functional as F

import nha_b200

DEV = 'cuda'
TRAINED = ('q_swa', 'k_swa', 'q_gsa', 'k_gsa', 'v', 's', 'g')


def listed():
    return [
        # a 340M training layer at its training batch: the headline
        dict(name='train_batch', kind='train', B=16, T=2048, HQ=16, H=16, D=64, M=64, window=64, shift=0, dtype='bfloat16'),
        # the smallest training call: a unit-test sized model in fp32, where launches and host work are what counts
        dict(name='train_smallest', kind='train', B=1, T=256, HQ=4, H=4, D=64, M=32, window=64, shift=0, dtype='float32'),
        # fine-tuning of a grouped-query model, ragged length, window and slot memory disjoint as the hybrid models have them
        dict(name='train_grouped', kind='train', B=2, T=1999, HQ=32, H=8, D=128, M=64, window=127, shift=128, dtype='bfloat16'),
        # packed training: ragged sequences, windows of 32 to 512 keys
        dict(name='train_packed', kind='packed', tokens=32768, shortest=128, longest=8192, pack=7, HQ=16, H=16, D=64, M=64),
        # a document of 128 K tokens, the long end of prefill
        dict(name='prefill_document', kind='prefill', B=1, T=131072, HQ=32, H=8, D=128, M=64, W=512, state=False, dtype='bfloat16'),
        # an ordinary chat prompt
        dict(name='prefill_prompt', kind='prefill', B=1, T=777, HQ=32, H=4, D=128, M=64, W=512, state=False, dtype='bfloat16'),
        # the next turn of several chats: slot memory handed in, seven query heads to a kv head
        dict(name='prefill_turn', kind='prefill', B=4, T=500, HQ=28, H=4, D=128, M=64, W=64, state=True, dtype='bfloat16'),
        # batched serving of a 48-layer model: 32 sequences a GPU
        dict(name='decode_batch', kind='decode', layers=48, B=32, HQ=32, H=4, D=128, M=64, W=512, state='float32'),
        # one user, a 24-layer small model: all launches and host work
        dict(name='decode_single', kind='decode', layers=24, B=1, HQ=16, H=16, D=64, M=64, W=64, state='float32'),
        # batched serving on the ring cache
        dict(name='decode_ring', kind='ring', layers=8, B=32, HQ=32, H=8, D=128, M=64, W=512),
        # the training layer's own inference step, window logits computed by the caller
        dict(name='recurrent_step', kind='recurrent', B=64, HQ=16, H=16, D=64, M=64, W=64),
        # the element-wise work of a 340M training layer around the operator
        dict(name='around_layer', kind='around', tokens=32768, H=16, D=64, M=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(('train', 'train', 'packed', 'prefill', 'prefill', 'decode', 'decode', 'ring', 'recurrent', 'around'))
    if kind == 'train':
        HQ, H, D = rng.choice(((4, 4, 64), (8, 8, 64), (16, 16, 64), (16, 16, 64), (16, 4, 64), (16, 16, 128), (32, 8, 128), (8, 2, 128)))
        M = rng.choice((64, 64, 64, 32))
        most = (1 << 25 if M == 64 else 1 << 21) // (HQ * D)
        tokens = _log(rng, 256, most)
        B = min(16, _log(rng, 1, max(1, tokens // 128)))
        window, shift = rng.choice(((64, 0), (63, 64), (32, 0), (127, 128), (256, 0)))
        return dict(kind=kind, B=B, T=max(1, tokens // B), HQ=HQ, H=H, D=D, M=M, window=window, shift=shift,
                    dtype=rng.choice(('bfloat16', 'bfloat16', 'bfloat16', 'float32')))
    if kind == 'packed':
        HQ, H, D = rng.choice(((8, 8, 64), (16, 16, 64), (16, 16, 64), (16, 4, 64), (8, 8, 128)))
        return dict(kind=kind, tokens=_log(rng, 2048, (1 << 25) // (HQ * D)), shortest=rng.choice((1, 16, 128)), longest=_log(rng, 600, 8192),
                    pack=rng.randrange(1 << 20), HQ=HQ, H=H, D=D, M=64)
    if kind == 'prefill':
        HQ, H, D, M = rng.choice(((16, 16, 64, 64), (8, 2, 64, 64), (32, 8, 128, 64), (32, 8, 128, 64), (32, 4, 128, 64), (28, 4, 128, 64), (8, 2, 64, 32)))
        dtype = rng.choice(('bfloat16', 'bfloat16', 'bfloat16', 'bfloat16', 'float32'))
        most = (1 << 28 if dtype == 'bfloat16' else 1 << 26) // (HQ * D)
        tokens = _log(rng, 200, min(most, 8192) if M == 32 or HQ // H == 7 else most)
        B = min(16, _log(rng, 1, max(1, tokens // 200)))
        return dict(kind=kind, B=B, T=tokens // B, HQ=HQ, H=H, D=D, M=M, W=rng.choice((32, 64, 64, 100, 128, 512)), state=rng.random() < 0.3, dtype=dtype)
    if kind in ('decode', 'ring'):
        HQ, H, D = rng.choice(((16, 16, 64), (8, 2, 64), (32, 8, 128), (32, 4, 128), (28, 4, 128)))
        W = rng.choice((64, 64, 128, 512, 300))
        layers = rng.choice((16, 24, 48)) if kind == 'decode' else rng.choice((4, 8))
        most = 48 * 32 * 4 * 128 * (64 * 8 + 512 * 2) // (layers * H * D * (64 * 8 + W * 2))
        c = dict(kind=kind, layers=layers, B=_log(rng, 1, max(1, min(most, 64))), HQ=HQ, H=H, D=D, M=64, W=W)
        if kind == 'decode':
            c['state'] = rng.choice(('float32', 'float32', 'float32', 'bfloat16'))
        return c
    if kind == 'recurrent':
        HQ, H, D = rng.choice(((16, 16, 64), (8, 2, 64), (32, 8, 128), (32, 4, 128)))
        return dict(kind=kind, B=_log(rng, 1, 256), HQ=HQ, H=H, D=D, M=rng.choice((64, 64, 32)), W=rng.choice((32, 64)))
    return dict(kind=kind, tokens=_log(rng, 200, 32768), H=rng.choice((8, 16, 32)), D=64, M=64)


# ---- inputs ----------------------------------------------------------------------------------------------------------

class _Source:
    """Values of one seed, made on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, scale=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=self.g, device=DEV) * scale).to(dtype)

    def gates(self, *shape, divided_by=1.0, dtype=torch.bfloat16):
        """Log forget gates and write weights of gate logits ~ N(0, 1)."""
        g = (F.logsigmoid(torch.randn(*shape, generator=self.g, device=DEV)) / divided_by).to(dtype)
        return g, (1 - g.float().exp()).to(dtype)


def _lengths(case):
    """Lengths and windows of the packed sequences."""
    r, lens = random.Random(case['pack']), []
    while sum(lens) < case['tokens']:
        lens.append(min(r.randint(case['shortest'], case['longest']), case['tokens'] - sum(lens)))
    return lens, [r.choice((32, 64, 128, 256, 512)) for _ in lens]


def _tables(positions, D):
    """Rotary tables [len(positions), D], halves duplicated."""
    inv = 1.0 / (10000.0 ** (torch.arange(0, D, 2, dtype=torch.float32, device=DEV) / D))
    a = torch.outer(torch.arange(*positions, dtype=torch.float32, device=DEV), inv)
    a = torch.cat([a, a], -1)
    return a.cos().bfloat16(), a.sin().bfloat16()


def prepare(case, seed):
    src, kind = _Source(seed), case['kind']
    s = dict(case=case)
    if kind in ('train', 'packed'):
        HQ, H, D, M = case['HQ'], case['H'], case['D'], case['M']
        dt = getattr(torch, case.get('dtype', 'bfloat16'))
        B, T = (case['B'], case['T']) if kind == 'train' else (1, case['tokens'])
        x = {n: src.normal(B, T, HQ if n[0] == 'q' else H, D, scale=D ** -0.5, dtype=dt) for n in TRAINED[:5]}
        x['g'], x['s'] = src.gates(B, T, H, M, dtype=dt)
        s['x'] = [x[n].requires_grad_(True) for n in TRAINED]
        s['do'] = src.normal(B, T, HQ, D, dtype=dt)
        if kind == 'train':
            s['how'] = dict(window_size_left=case['window'], window_size_right=0, gsa_kv_shift=case['shift'])
        else:
            lens, windows = _lengths(case)
            ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
            s['how'] = dict(cu_seqlens=ints([sum(lens[:i]) for i in range(len(lens) + 1)]), max_seqlen=max(lens), window_size_left=ints(windows),
                            window_size_right=0, gsa_kv_shift=0)
    elif kind == 'prefill':
        B, T, HQ, H, D, M = (case[n] for n in ('B', 'T', 'HQ', 'H', 'D', 'M'))
        dt = getattr(torch, case['dtype'])
        g, w = src.gates(B, T, H, M, divided_by=8.0, dtype=dt)
        s['how'] = dict(q=src.normal(B, T, HQ, D, dtype=dt), rotary_q=src.normal(B, T, HQ, D, dtype=dt), k=src.normal(B, T, H, D, dtype=dt),
                        rotary_k=src.normal(B, T, H, D, dtype=dt), v=src.normal(B, T, H, D, dtype=dt), s=w, g=g, window_size=case['W'],
                        output_final_state=True)
        if case['state']:
            s['how']['initial_state'] = (src.normal(B, H, D, M, scale=0.5, dtype=torch.float32), src.normal(B, H, M, D, scale=0.5, dtype=torch.float32))
    elif kind in ('decode', 'ring'):
        L, B, HQ, H, D, M, W = (case[n] for n in ('layers', 'B', 'HQ', 'H', 'D', 'M', 'W'))
        q, k, v = src.normal(L, B, 1, HQ, D), src.normal(L, B, 1, H, D), src.normal(L, B, 1, H, D)
        g, _ = src.gates(L, B, 1, H, M, divided_by=8.0)
        dt = getattr(torch, case.get('state', 'float32'))
        hk, hv = src.normal(L, B, H, D, M, scale=0.5, dtype=dt), src.normal(L, B, H, M, D, scale=0.5, dtype=dt)
        cos, sin = (t[None] for t in _tables((32769 - W, 32769), D))
        win_k, win_v = src.normal(L, B, W, H, D), src.normal(L, B, W, H, D)
        if kind == 'decode':
            s.update(hk=hk, hv=hv, layers=[dict(q=q[i], k=k[i], v=v[i], g=g[i], sw_k=win_k[i], sw_v=win_v[i], cos=cos, sin=sin,
                                                initial_state=(hk[i], hv[i]), output_final_state=True) for i in range(L)])
        else:
            win_g, _ = src.gates(L, B, W, H, M, divided_by=8.0)
            s['cache'] = nha_b200.NHARingCache()
            for i in range(L):
                s['cache'].init_layer(i, win_k[i], win_v[i], win_g[i], W, (hk[i], hv[i]))
            s['layers'] = [(i, q[i], k[i], v[i], g[i], cos, sin) for i in range(L)]
    elif kind == 'recurrent':
        B, HQ, H, D, M, W = (case[n] for n in ('B', 'HQ', 'H', 'D', 'M', 'W'))
        g, w = src.gates(B, 1, H, M, divided_by=8.0)
        s['how'] = dict(q=src.normal(B, 1, HQ, D), k=src.normal(B, 1, H, D), v=src.normal(B, 1, H, D), sliding_window=src.normal(B, 1, HQ, W), s=w, g=g,
                        initial_state=(src.normal(B, H, D, M, scale=0.5, dtype=torch.float32), src.normal(B, H, M, D, scale=0.5, dtype=torch.float32)),
                        output_final_state=True)
    else:
        T, H, D, M = (case[n] for n in ('tokens', 'H', 'D', 'M'))
        s['x'] = [src.normal(1, T, H, n).requires_grad_(True) for n in (D, D, D, M)] + [src.normal(1, T, H * D).requires_grad_(True)]
        s['lse'] = [src.normal(1, T, H, scale=3.0, dtype=torch.float32), src.normal(1, T, H, scale=3.0, dtype=torch.float32).requires_grad_(True)]
        s['weight'] = (torch.rand(H * D, generator=src.g, device=DEV) + 0.5).requires_grad_(True)
        s['cos'], s['sin'] = (t[:, :D // 2].contiguous() for t in _tables((T,), D))
        s['up'] = [src.normal(1, T, H, n) for n in (D, D, D, D, D, M, M)] + [src.normal(1, T, H * D), torch.ones((), device=DEV)]
    return s


# ---- one pass --------------------------------------------------------------------------------------------------------

def run(state):
    kind = state['case']['kind']
    if kind in ('train', 'packed'):
        o, lse_swa, lse_gsa = nha_b200.chunk_nha(*state['x'], **state['how'])
        return [o.detach(), lse_swa, lse_gsa.detach(), *torch.autograd.grad(o, state['x'], state['do'])]
    if kind == 'prefill':
        return nha_b200.fused_chunk_nha_prefill(**state['how'])
    if kind == 'decode':
        step = nha_b200.fused_recurrent_nha_decode
        if state['hk'].dtype == torch.bfloat16:
            step = nha_b200.fused_recurrent_nha_decode_bf16_state
        return [step(**layer)[0] for layer in state['layers']] + [state['hk'], state['hv']]
    if kind == 'ring':
        cache = state['cache']
        out = [cache.decode(*layer) for layer in state['layers']]
        return [(o, y.hk, y.hv, y.ring_k, y.ring_v, y.ring_g, y.head) for o, y in zip(out, cache)]
    if kind == 'recurrent':
        return nha_b200.fused_recurrent_nha(**state['how'])
    q, k, v, f, o = state['x']
    front = [*nha_b200.feature_maps(q, k, v), *nha_b200.rotary_pair(q, k, state['cos'], state['sin']), *nha_b200.slot_gates(f)]
    y = nha_b200.silu_rms_norm(o, state['weight'])
    loss, share = nha_b200.gsa_aux_loss(*state['lse'], 0.3)
    grads = torch.autograd.grad([*front, y, loss], [*state['x'], state['weight'], state['lse'][1]], state['up'])
    return [*(t.detach() for t in (*front, y, loss, share)), *grads]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def _keys(T, left):
    """Window keys that the queries of a sequence of T tokens see together."""
    full = max(0, T - left)
    return full * (left + 1) + (T - full) * (T - full + 1) // 2


def work(case):
    kind, D = case['kind'], case['D']
    H, M = case['H'], case['M']
    HQ = case.get('HQ', H)
    wide = 4 if case.get('dtype') == 'float32' else 2
    if kind in ('train', 'packed', 'prefill'):
        if kind == 'packed':
            lens, left = _lengths(case)
            N, T = len(lens), sum(lens)
            keys = sum(_keys(n, w) for n, w in zip(lens, left))
        else:
            N, T = case['B'], case['B'] * case['T']
            keys = N * _keys(case['T'], case['window'] if kind == 'train' else case['W'] - 1)
        # slot memory read by every query and written by every key, window keys by every query that sees them
        flops = T * HQ * 4 * D * M + T * H * 4 * D * M + keys * HQ * 4 * D
        once = T * (2 * HQ * D + 3 * H * D + 2 * H * M) * wide                  # q, k of both branches, v, s, g
        if kind == 'prefill':
            return dict(bytes=once + T * HQ * D * wide + N * H * 2 * D * M * 4 * (2 if case['state'] else 1), flops=flops)
        # the backward has two products for each one of the forward; its gradients, do, o and the log-sum-exps
        return dict(bytes=2 * once + 2 * T * HQ * D * wide + T * HQ * 8, flops=3 * flops)
    if kind in ('decode', 'ring'):
        L, B, W = case['layers'], case['B'], case['W']
        size = 4 if case.get('state', 'float32') == 'float32' else 2
        window = B * W * H * 2 * D * 2
        step = B * (2 * HQ * D + H * (2 * D + M)) * 2 * (1 if kind == 'decode' else 2)
        return dict(bytes=L * (window + 2 * B * H * 2 * D * M * size + step), flops=L * B * (HQ * 4 * D * (M + W) + H * 4 * D * M))
    if kind == 'recurrent':
        B, W = case['B'], case['W']
        return dict(bytes=2 * B * H * 2 * D * M * 4 + B * (HQ * (2 * D + W) + H * (2 * D + 2 * M)) * 2 + B * HQ * W * 4,
                    flops=B * (HQ * 4 * D * M + H * 4 * D * M))
    T = case['tokens']
    # q, k, v, gates, o in; their eight results out; upstream gradients in; gradients out; the log-sum-exps
    return dict(bytes=2 * T * H * ((3 * D + M + D) + (3 * D + 2 * D + 2 * M + D) * 2 + (3 * D + M + D)) + T * H * 12, flops=T * H * D * 60)


def tolerance(case):
    kind = case['kind']
    if kind in ('train', 'packed'):
        # gradients are chains of products whose operands are rounded to bf16, and the one of the gates is a difference of
        # large terms: the tensor-core and the general kernels, both correct, are 2.9e-2 apart there (5e-3 elsewhere)
        return dict(rel=3e-2)
    return dict(rel=1e-2)
