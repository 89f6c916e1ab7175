"""The fp16-query decode-attention kernel against 64-bit arithmetic over the rows the store holds: group sizes on both sides of
the halved softmax, tile and bucket edges, widths alone and mixed, and more runs than a CTA handles between two merges."""
import math

import numpy as np
import pytest
import torch

from oracle import smartkv_oracle as orc
from smartkv_b200 import _lib
from tests.gpu_util import fill_store, make_store

pytestmark = pytest.mark.gpu


def check(hq, hkv, d, n, batch, widths, seed, sequences=None, masked=False, value_gain=None, plan_of_128=False):
    rng = np.random.default_rng(seed)
    k, v = orc.synth_kv(batch * n, hkv, d, seed=seed)
    if value_gain is not None:
        v = (v * rng.uniform(*value_gain, size=(batch * n, hkv, 1))).astype(np.float32)
    bits = rng.choice(widths, size=(batch, n))
    store = make_store(1, batch, hkv, d, hq, n)
    fill_store(store, [(k.reshape(batch, n, hkv, d), v.reshape(batch, n, hkv, d))], bits)
    q = torch.from_numpy(rng.standard_normal((batch, hq, d)).astype(np.float16)).cuda()
    mask = None
    if masked:      # single keys, whole tiles of 16 and beyond, and ordinary values
        mask = torch.from_numpy(rng.standard_normal((batch, n)).astype(np.float32)).cuda()
        mask[:, 5::11] = -1e4
        mask[:, n // 3:n // 2] = float("-inf")
    if plan_of_128:
        _lib.lib().skv_set_attention_path(2)
        try:
            store.build_plan()
        finally:
            _lib.lib().skv_set_attention_path(0)
        assert int(store.plan[3]) == 128 and store._plan_valid
    out = store.attention(0, q, mask=mask).double()
    store.check_errors()
    group = hq // hkv
    for b in sequences or range(batch):
        ids, _, kc, vc, ks, vs = store.export_sequence(0, b)
        bias = 0.0 if mask is None else mask[b, ids.long()].double()
        for h in range(hkv):
            kd, vd = kc[:, h].double() * ks[:, h, None].double(), vc[:, h].double() * vs[:, h, None].double()
            qd = q[b, h * group:(h + 1) * group].double()
            p = torch.softmax(qd @ kd.T / math.sqrt(d) + bias, -1)
            # p * v_scale is rounded to fp16 (2^-11 of each term); the query to 2^-15 of its row's largest element, which moves
            # a logit by at most that times sum |k| / sqrt(d) and a probability by twice as much of itself
            logit = qd.abs().amax(1, keepdim=True) * 2.0 ** -15 * kd.abs().sum(1).max() / math.sqrt(d)
            bound = (2.0 ** -11 + 2 * logit) * (p @ vd.abs()) + 1e-6
            err = (out[b, h * group:(h + 1) * group] - p @ vd).abs()
            assert bool((err <= bound).all()), (b, h, float((err / bound).max()))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("group", [1, 3, 4, 5, 8])
def test_group_sizes(d, group):
    check(2 * group, 2, d, 203, 2, (2, 3, 4, 8), seed=group + d)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("width", [2, 3, 4, 8])
@pytest.mark.parametrize("n", [1, 17, 4096 + 5])
def test_one_width(d, width, n):
    check(8, 2, d, n, 1, (width,), seed=n + width)


# 2 x 2 x 331 keys are a tile or less a warp; one sequence of 40007 keys gives every warp several, with a ragged last one
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("group", [4, 5, 8])
@pytest.mark.parametrize("hkv,n,batch", [(2, 331, 2), (1, 40007, 1)])
def test_masked(d, group, hkv, n, batch):
    check(group * hkv, hkv, d, n, batch, (2, 3, 4, 8), seed=group + n, masked=True)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("group", [4, 8])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("hkv,n,batch", [(2, 331, 2), (1, 40007, 1)])
def test_value_scales_beyond_the_fp16_guard(d, group, masked, hkv, n, batch):
    # scales of 10 to 1e5: some below the limit of 64 and most above it, so the running maximum is raised for some tiles
    check(group * hkv, hkv, d, n, batch, (2, 3, 4, 8), seed=group + n, masked=masked, value_gain=(10, 1e5))


@pytest.mark.parametrize("group", [4, 8])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("hkv,n,batch", [(2, 331, 2), (1, 40007, 1)])
def test_plan_in_tiles_of_128_keys(group, masked, hkv, n, batch):
    check(group * hkv, hkv, 128, n, batch, (2, 3, 4, 8), seed=group + n, masked=masked, plan_of_128=True)


def test_one_long_segment_over_all_ctas():
    check(8, 1, 128, 40007, 1, (2, 3, 4, 8), seed=5)


def test_more_runs_than_a_merge_holds():
    # 1600 segments: eleven or so in each of 148 CTAs, eight between two merges
    check(32, 8, 128, 21, 200, (2, 3, 4, 8), seed=6, sequences=(0, 1, 73, 199))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("group", [4, 8])
@pytest.mark.parametrize("masked_with", [float("-inf"), float(torch.finfo(torch.float32).min)])
@pytest.mark.parametrize("width", [2, 8])
def test_warps_that_hold_only_masked_infinite_values_do_not_count(d, group, masked_with, width):
    """Three tiles for every CTA, one for each of three warps: every third tile's keys are masked and their V rows infinite.  The
    warps are folded by weight, and those of weight 0 hold NaN."""
    n = 16 * 148 * 3
    gen = torch.Generator(device="cuda").manual_seed(d + group)
    store = make_store(1, 1, 1, d, group, n)
    k, v = (torch.randn((n, 1, d), generator=gen, device="cuda") for _ in range(2))
    hidden = torch.arange(n, device="cuda") % 48 < 16
    v[hidden, 0, 5] = float("inf")
    dst = store.plan_bulk(torch.full((1, n), width, dtype=torch.int64, device="cuda"))
    store.append(0, k, v, *dst[:3])
    q = torch.randn((1, group, d), generator=gen, device="cuda").half()
    mask = torch.zeros((1, n), device="cuda")
    mask[0, hidden] = masked_with
    out = store.attention(0, q, mask=mask).double()[0]
    store.check_errors()
    _, _, kc, vc, ks, vs = store.export_sequence(0, 0)
    seen = ~hidden
    kd, vd = kc[seen, 0].double() * ks[seen].double(), vc[seen, 0].double() * vs[seen].double()
    p = torch.softmax(q[0].double() @ kd.T / math.sqrt(d), -1)
    logit = q[0].double().abs().amax(1, keepdim=True) * 2.0 ** -15 * kd.abs().sum(1).max() / math.sqrt(d)
    bound = (2.0 ** -11 + 2 * logit) * (p @ vd.abs()) + 1e-6    # as in check()
    assert bool(((out - p @ vd).abs() <= bound).all())


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("group", [4, 8])
def test_the_weight_of_a_key_far_above_all_before_it_is_not_rounded(d, group):
    """One CTA, four tiles a warp.  One key stands 2^4.5 to 2^7.5 above the others, in the last tile of the first warp; the
    others have no value.  Its row is 2 bits wide, so its V scale is the fp16 number it was made from, and once it sets the
    running maximum its weight times that scale is exact: what is left is 32-bit arithmetic.  Rounded to fp16 the weight would
    be off by up to 2^-11."""
    n = 16 * 4 * (16 if d == 64 else 12)
    at = 16 * 3 + 5
    store = make_store(1, 1, 1, d, group, n)
    store.num_ctas = 1
    k, v = torch.zeros((n, 1, d), device="cuda"), torch.zeros((n, 1, d), device="cuda")
    k[at, 0, 7] = 1.0
    v[at, 0] = torch.where(torch.arange(d, device="cuda") % 3 == 0, 0.7, -0.7).half().float()
    dst = store.plan_bulk(torch.full((1, n), 2, dtype=torch.int64, device="cuda"))
    store.append(0, k, v, *dst[:3])
    above = torch.linspace(4.5, 7.5, group, device="cuda", dtype=torch.float64)
    q = torch.zeros((1, group, d), device="cuda", dtype=torch.float16)
    q[0, :, 7] = (above * math.sqrt(d) * math.log(2.0)).half()
    out = store.attention(0, q).double()[0]
    store.check_errors()
    p = torch.softmax(torch.where(torch.arange(n, device="cuda") == at, q[0, :, 7:8].double() / math.sqrt(d), 0.0), -1)
    ref = p[:, at:at + 1] * v[at, 0].double()
    # the query's one element is a whole number of limb steps, so the logit (at most 7.5 log2 units) and the sum of up to 1024
    # weights carry 32-bit roundings only: 2^-16 leaves room for 2^8 of them
    assert bool(((out - ref).abs() <= 2.0 ** -16 * ref.abs()).all())
