"""GPU: an odd number of query heads per kv head in the tensor-memory output passes (the last 128-row tile of a group holds
one head), against the oracle: ragged last chunk, the last group of the tensor (nothing behind it), initial state."""
import pytest

from oracle import nha_oracle as orc
from tests import inputs as gen
from tests.gpu_util import TOL_OUT, assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('K,NG,W,T,state', [(128, 7, 64, 130, True), (128, 3, 200, 300, False), (128, 1, 64, 70, True),
                                            (64, 7, 64, 130, True), (64, 3, 200, 257, False)])
def test_prefill_with_odd_groups(K, NG, W, T, state):
    from nha_b200 import fused_chunk_nha_prefill
    d = gen.prefill_inputs(300 + K + NG, 2, 2, NG, K, K, 64, W, T, with_state=state)
    want = orc.prefill(d['q'], d['k'], d['v'], d['rotary_q'], d['rotary_k'], d['s'], d['g'], W, d['scale'], d.get('hk0'), d.get('hv0'))
    c = {n: x.cuda() if hasattr(x, 'cuda') else x for n, x in d.items()}
    o, (hk, hv) = fused_chunk_nha_prefill(q=c['q'], k=c['k'], v=c['v'], rotary_q=c['rotary_q'], rotary_k=c['rotary_k'], s=c['s'], g=c['g'],
                                          window_size=W, output_final_state=True,
                                          initial_state=(c['hk0'], c['hv0']) if state else None)
    for got, ref, name in zip((o, hk, hv), want, ('o', 'hk', 'hv')):
        assert_close(got, ref, TOL_OUT, name)
