"""GPU: the merge of a (sequence, kv head) that several CTAs share in the streaming decode kernel, through the cluster and through the workspace."""
import pytest
import torch

from oracle import nha_oracle as orc
from tests import inputs as gen
from tests.gpu_util import TOL_OUT, assert_close, cuda

pytestmark = pytest.mark.gpu


# two, four, eight and sixteen CTAs; one head, a group that fills its lanes, an odd one, and one that takes two rounds of threads
@pytest.mark.parametrize('NG', [1, 4, 7, 16])
@pytest.mark.parametrize('D,W', [(64, 256), (128, 256), (64, 512), (128, 520), (64, 1200), (128, 1200), (128, 2100)])
def test_merges_against_the_oracle(D, W, NG, monkeypatch):
    from nha_b200 import fused_recurrent_nha_decode
    B, H, M = 2, 2, 64
    d = gen.decode_inputs(40 + W + NG, B, H, NG, D, D, M, W)
    d['cos'], d['sin'] = gen.rope_tables(W, D, first_pos=3000)
    ref = orc.decode_step(d['q'], d['k'], d['v'], d['g'], d['sw_k_raw'], d['vw'], d['scale'], cos=d['cos'], sin=d['sin'], hk0=d['hk0'], hv0=d['hv0'])
    c, out = cuda(d), []
    for off in ('0', '1'):
        monkeypatch.setenv('NHA_B200_DECODE_NO_CLUSTER', off)
        o, (hk, hv) = fused_recurrent_nha_decode(q=c['q'], k=c['k'], v=c['v'], g=c['g'], sw_k=c['sw_k_raw'], sw_v=c['vw'], cos=c['cos'], sin=c['sin'],
                                                 initial_state=(c['hk0'].clone(), c['hv0'].clone()), output_final_state=True)
        assert_close(o, ref[0], TOL_OUT, f'o, workspace {off}')
        assert_close(hk, ref[1], 1e-5, 'hkt')
        assert_close(hv, ref[2], 1e-5, 'hvt')
        out.append(o.float())
    # the same fp32 partial results: at most one step of the bf16 result apart
    assert torch.allclose(*out, rtol=2.0 ** -7, atol=1e-6)
