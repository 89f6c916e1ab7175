"""skv_importance_update over head counts, bucket fills, array alignments and sizes on both sides of the limit between one and four
storage indices a thread: the same bits in every form, and the 64-bit sums within the rounding of 32-bit ones."""
import ctypes

import pytest
import torch

from smartkv_b200 import _lib
from smartkv_b200._lib import check, ptr
from smartkv_b200.store import PackedKVStore

pytestmark = pytest.mark.gpu


def shifted(t, elements):
    """A copy of t whose storage starts `elements` behind an aligned address."""
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    out = buf[elements:elements + t.numel()].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("heads", [1, 8, 9, 32, 128])
@pytest.mark.parametrize("counts", [(0, 0, 0, 0), (1, 3, 127, 5), (128, 0, 126, 1023), (1021, 130, 2, 64)])
@pytest.mark.parametrize("batch", [3, 66])
def test_importance_update(heads, counts, batch):
    # 2688 storage indices a sequence; up to 4 x 148 blocks of 256 take one a thread, 66 sequences are more
    layers, layer = 2, 1
    store = PackedKVStore(layers, batch, 1, 64, 8, (1152, 256, 128, 1152))
    slots = store.slots
    assert (batch * slots <= 4 * 148 * 256) == (batch == 3)
    gen = torch.Generator(device="cuda").manual_seed(heads)
    rand = lambda *s: torch.rand(s, generator=gen, device="cuda")
    filled = torch.tensor([counts, (0, 0, 0, 0), counts] * (batch // 3), dtype=torch.int32, device="cuda")
    base = store.bucket_base
    cur_slot = torch.tensor([base[2] + counts[2] if counts[2] < 128 else base[0] + counts[0], base[3], -1] * (batch // 3),
                            dtype=torch.int32, device="cuda")
    logits, lse_max, lse_sum = -8 * rand(batch, heads, slots), rand(batch, heads), 1 + 9 * rand(batch, heads)
    cur_prob, head_state = rand(batch, heads), 0.5 + rand(batch, 2, heads)
    cumulative, ema = torch.rand((batch, slots), generator=gen, device="cuda", dtype=torch.float64), rand(layers, batch, slots)
    touched = (rand(layers, batch, slots) < 0.5).to(torch.uint8)
    decay, head_decay = 0.9, 0.8

    def update(desc, offset, *arrays):
        filled, lg, lse_max, lse_sum, cur_prob, cur_slot, hs, cm, em, tc = arrays
        lg, cm, em, tc, hs = (shifted(t, offset) for t in (lg, cm, em, tc, hs))
        check(store.lib.skv_importance_update(ctypes.byref(desc), layer, ptr(filled), heads, ptr(lg), ptr(lse_max), ptr(lse_sum),
                                              ptr(cur_prob), ptr(cur_slot), ptr(hs), 0, ptr(cm), ptr(em), ptr(tc), decay, head_decay,
                                              _lib.stream_ptr()))
        return cm, em, tc, hs

    arrays = (filled, logits, lse_max, lse_sum, cur_prob, cur_slot, head_state, cumulative, ema, touched)
    results = [update(store.desc, offset, *arrays) for offset in (0, 1)]
    for a, b in zip(*results):
        assert torch.equal(a, b)
    alone = PackedKVStore(layers, 1, 1, 64, 8, (1152, 256, 128, 1152)).desc
    for b in range(3):      # a sequence by itself takes one index a thread
        one = update(alone, 0, *(t[:, b:b + 1].contiguous() if t is ema or t is touched else t[b:b + 1].contiguous() for t in arrays))
        cm, em, tc, hs = results[0]
        for x, y in zip(one, (cm[b:b + 1], em[:, b:b + 1], tc[:, b:b + 1], hs[b:b + 1])):
            assert torch.equal(x, y)
    cm, em, tc, hs = results[0]
    want_c, want_e, want_t = cumulative.clone(), ema.double(), touched.clone()
    for b in range(batch):
        total = int(filled[b].sum()) + int(cur_slot[b] >= 0)
        hn = head_state[b, 0].double() * head_decay + (1 - head_decay) * (1.0 / total if total else 0.0)
        assert torch.allclose(hs[b, 1].double(), hn, rtol=1e-6)
        w = hn / (hn.mean() + 1e-6)
        keys = [base[i] + k for i in range(4) for k in range(int(filled[b, i]))]
        mass = (w[:, None] * torch.exp2(logits[b].double() - lse_max[b].double()[:, None]) / lse_sum[b].double()[:, None]).sum(0)
        if cur_slot[b] >= 0:
            keys.append(int(cur_slot[b]))
            mass[cur_slot[b]] = (w * cur_prob[b].double()).sum()
        if not keys:
            continue
        i = torch.tensor(keys, device="cuda")
        want_c[b, i] += mass[i]
        want_e[layer, b, i] = torch.where(touched[layer, b, i] > 0, decay * want_e[layer, b, i] + (1 - decay) * mass[i], mass[i])
        want_t[layer, b, i] = 1
    # a sum of `heads` products in 32 bits, each exponential good to 2^-22
    rtol = (heads + 8) * 2.0 ** -23
    assert torch.allclose(cm, want_c, rtol=rtol, atol=0) and torch.allclose(em.double(), want_e, rtol=rtol, atol=0)
    assert torch.equal(tc, want_t)
