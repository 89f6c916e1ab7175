"""The combine over segments of few and of many partials, for every kernel that leaves them (fp16 queries: one partial a run; fp32
queries: seven; tensor memory: four): remainders of the rows it has in flight, the edge of a chunk of 256, several chunks."""
import math

import pytest
import torch

from oracle import smartkv_oracle as orc
from smartkv_b200 import _lib
from tests.gpu_util import fill_store, make_store

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 3, 36, 37, 64, 65, 148])   # partials: 2..149; 7, 21, 252, 259, 448, 455, 1036; 4, 12, 144, ...
@pytest.mark.parametrize("kernel,d", [("f16", 64), ("f16", 128), ("f32", 64), ("f32", 128), ("tensor_memory", 128)])
def test_one_segment_over_some_ctas(kernel, d, ctas):
    group, n = 4, 148 * 128 + 5
    store = make_store(1, 1, 1, d, group, n)
    store.num_ctas = ctas
    gen = torch.Generator(device="cuda").manual_seed(ctas + d)
    bits = torch.tensor([2, 3, 4, 8], device="cuda")[torch.randint(4, (1, n), generator=gen, device="cuda")]
    k, v = orc.synth_kv(n, 1, d, seed=ctas)
    fill_store(store, [(k[None], v[None])], bits.cpu().numpy())
    q = torch.randn((1, group, d), generator=gen, device="cuda")
    q = q if kernel == "f32" else q.half()
    cur_k, cur_v = (torch.randn((1, 1, d), generator=gen, device="cuda") for _ in range(2))
    try:
        _lib.lib().skv_set_attention_path(2 if kernel == "tensor_memory" else 0)
        out = store.attention(0, q, cur_k, cur_v).double()[0]
        store.check_errors()
    finally:
        _lib.lib().skv_set_attention_path(0)
    _, _, kc, vc, ks, vs = store.export_sequence(0, 0)
    kd = torch.cat([kc[:, 0].double() * ks.double(), cur_k[0].double()])
    vd = torch.cat([vc[:, 0].double() * vs.double(), cur_v[0].double()])
    qd = q[0].double()
    p = torch.softmax(qd @ kd.T / math.sqrt(d), -1)
    # fp16: p * v_scale to 2^-11, the query to 2^-15 of its largest element (which moves a probability by twice the logit's
    # error); fp32: the weight in two such halves, of which the lower may be below fp16's normal range (2^-16 of the sum then),
    # the query in three limbs
    weight, limb = (2.0 ** -16, 2.0 ** -22) if kernel == "f32" else (2.0 ** -11, 2.0 ** -15)
    logit = qd.abs().amax(1, keepdim=True) * limb * kd.abs().sum(1).max() / math.sqrt(d)
    bound = (weight + 2 * logit) * (p @ vd.abs()) + 1e-6
    err = (out - p @ vd).abs()
    assert bool((err <= bound).all()), float((err / bound).max())
