"""Fused importance update vs the oracle's restatement of update_attention."""
import numpy as np
import pytest
import torch

from oracle import smartkv_oracle as orc
from tests.gpu_util import assert_close, fill_store, make_store, oracle_attention, oracle_quantized

pytestmark = pytest.mark.gpu


def test_importance_over_steps_and_layers():
    hq, hkv, d, n0, Lyr, B, steps = 16, 4, 64, 150, 2, 2, 3
    g = hq // hkv
    rng = np.random.default_rng(5)
    store = make_store(Lyr, B, hkv, d, hq, n0 + steps + 1)
    bits = rng.choice([2, 3, 4, 8], size=(B, n0))
    kv = []
    for layer in range(Lyr):
        ks, vs = zip(*[orc.synth_kv(n0, hkv, d, seed=40 + 10 * layer + b) for b in range(B)])
        kv.append((np.stack(ks), np.stack(vs)))
    fill_store(store, kv, bits)
    # oracle state: one per sequence (the reference keeps one cache per sequence)
    ostate = [orc.ImportanceState(Lyr) for _ in range(B)]
    cache = [[list(oracle_quantized(kv[l][0][b], kv[l][1][b], bits[b])) for l in range(Lyr)] for b in range(B)]
    for step in range(steps):
        plan = store.plan_step()
        for layer in range(Lyr):
            q = rng.standard_normal((B, hq, d)).astype(np.float32)
            ck = rng.standard_normal((B, hkv, d)).astype(np.float32)
            cv = rng.standard_normal((B, hkv, d)).astype(np.float32)
            store.attention(layer, torch.from_numpy(q).cuda(), torch.from_numpy(ck).cuda(), torch.from_numpy(cv).cuda(),
                            update_importance=True, cur_storage=plan[3])
            store.append(layer, torch.from_numpy(ck).cuda(), torch.from_numpy(cv).cuda(), plan[0], plan[1], plan[2])
            for b in range(B):
                kq, vq, ks, vs = cache[b][layer]
                _, p = oracle_attention(q[b], kq, vq, ks, vs, g, ck[b], cv[b])
                ostate[b].update(layer, p[None, :, None, :], list(range(p.shape[-1])))
                nk, nv, nks, nvs = oracle_quantized(ck[b][None], cv[b][None], np.array([4]))
                cache[b][layer] = [np.concatenate([kq, nk]), np.concatenate([vq, nv]), np.concatenate([ks, nks]),
                                   np.concatenate([vs, nvs])]
        store.commit_step(plan)
    store.check_errors()
    st = store.slot_token.cpu().numpy()
    cum = store.cumulative.cpu().numpy()
    ema = store.layer_ema.cpu().numpy()
    n = n0 + steps
    for b in range(B):
        valid = st[b] >= 0
        assert valid.sum() == n
        order = np.argsort(st[b][valid])
        got = cum[b][valid][order]
        want = np.array([ostate[b].token_importance[t] for t in range(n)])
        assert_close(got, want, 1e-6, 2e-3, f"cumulative importance seq {b}")
        for layer in range(Lyr):
            got_l = ema[layer, b][valid][order]
            want_l = np.array([ostate[b].layer_importance[(layer, t)] for t in range(n)])
            assert_close(got_l, want_l, 1e-6, 2e-3, f"layer EMA seq {b} layer {layer}")
        hs = store.head_state.cpu().numpy()[b, store.head_parity]
        assert_close(hs, ostate[b].head_importance, 1e-7, 1e-5, "head importance EMA")
    # appended tokens landed in the 4-bit bucket and read back bit-exact
    for b in range(B):
        ids, wb, kc, vc, ks, vs = store.export_sequence(1, b)
        assert np.array_equal(wb.cpu().numpy()[n0:], np.full(steps, 4))
        assert np.array_equal(kc.cpu().numpy(), cache[b][1][0])
        assert np.array_equal(vs.cpu().numpy(), cache[b][1][3])


@pytest.mark.parametrize("B,n,first", [(1, 1, 0), (3, 130, 0), (2, 300, 299), (5, 257, 100)])
def test_token_places_and_prompt_importance(B, n, first):
    """Against index expressions over the store's own bookkeeping, tokens spread over all buckets, one more asked for than
    there are; the fp32 arithmetic is the same operation by operation, so the results are equal."""
    from tests.gpu_util import make_store
    g = torch.Generator(device="cuda").manual_seed(n)
    store = make_store(2, B, 2, 64, 4, n + 1)
    bits = torch.tensor([2, 3, 4, 8], device="cuda")[torch.randint(0, 4, (B, n), generator=g, device="cuda")]
    seq, bucket, pos, storage = store.plan_bulk(bits)
    count = n - first
    got = store.token_places(count + 1, torch.tensor([first], device="cuda"))
    for have, want in zip(got, (seq, bucket, pos, storage.to(torch.int32).view(-1))):
        assert torch.equal(have.view(B, -1)[:, :count], want.view(B, n)[:, first:])
    assert bool((got[0].view(B, -1)[:, count] == -1).all()) and bool((got[3].view(B, -1)[:, count] == -1).all())
    mass = [torch.rand((B, n), generator=g, device="cuda") for _ in range(3)]
    at = storage.long()
    store.cumulative.fill_(7.0)
    store.prompt_importance(0, mass[0], assign=True)
    store.prompt_importance(1, mass[1], assign=False)
    store.prompt_importance(1, mass[2], assign=False)
    assert torch.equal(store.cumulative.gather(1, at), (mass[0].double() + mass[1].double()) + mass[2].double())
    assert torch.equal(store.layer_ema[0].gather(1, at), mass[0])
    assert torch.equal(store.layer_ema[1].gather(1, at), store.decay * mass[1] + (1 - store.decay) * mass[2])
    assert int(store.touched.sum()) == 2 * B * n and int((store.cumulative != 7.0).sum()) == B * n
