"""GPU parity of quantize / pack / append against the CPU oracle: bit-exact."""
import ctypes
import hashlib

import numpy as np
import pytest
import torch

from oracle import smartkv_oracle as orc

pytestmark = pytest.mark.gpu


def _lib():
    from smartkv_b200 import _lib
    return _lib


def _quantize_gpu(x, bits):
    L = _lib()
    xt = torch.from_numpy(x).cuda().contiguous()
    rows = xt.numel() // xt.shape[-1]
    codes = torch.empty(xt.shape, dtype=torch.int8, device="cuda")
    scales = torch.empty(xt.shape[:-1], dtype=torch.float32, device="cuda")
    code = L.DTYPE_F32 if xt.dtype == torch.float32 else L.DTYPE_F16
    L.check(L.lib().skv_quantize_per_head(L.ptr(xt), code, rows, xt.shape[-1], bits, L.ptr(codes), L.ptr(scales),
                                          L.stream_ptr()))
    torch.cuda.synchronize()
    return codes.cpu().numpy(), scales.cpu().numpy()


@pytest.mark.parametrize("tag", ["a", "b"])
@pytest.mark.parametrize("bits", [2, 3, 4, 8])
def test_quantize_golden_bit_exact(golden, tag, bits):
    g = golden("quant")
    for name in ("k", "v"):
        q, s = _quantize_gpu(g[f"quant_{tag}_{name}"], bits)
        assert np.array_equal(q, g[f"quant_{tag}_{name}q{bits}"])
        assert np.array_equal(s.view(np.uint32), g[f"quant_{tag}_{name}s{bits}"].view(np.uint32))


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("d", [64, 128, 80])
def test_quantize_random_vs_oracle(bits, d):
    rng = np.random.default_rng(bits * 100 + d)
    x = (rng.standard_normal((777, d)) * rng.choice([1e-3, 1.0, 50.0], size=(777, 1))).astype(np.float32)
    x[5] = 0
    x[6, :] = np.round(x[6] * 4) / 4
    q, s = _quantize_gpu(x, bits)
    qo, so = orc.quantize_rows(x, bits)
    assert np.array_equal(q, qo)
    assert np.array_equal(s.view(np.uint32), so.view(np.uint32))


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("d", [64, 128])
def test_quantize_near_ties_and_extreme_scales(bits, d):
    """Values whose quotient x / scale sits on or next to a half-integer, and rows whose scale is
    tiny, huge or subnormal: the kernel's reciprocal-multiply shortcut must fall back to the IEEE
    division exactly where the two could round differently."""
    rng = np.random.default_rng(900 + bits + d)
    levels = max(2 ** (bits - 1) - 1, 1)
    rows = []
    for amax in (1.0, 3.0, 0.7310585, 127.0, 1e-3, 6.1e-5, 2.5e7, 1e-33, 1e33, 3e-39, 1e-44):
        amax = np.float32(amax)
        s = np.float32(amax / np.float32(levels))
        for _ in range(24):
            k = rng.integers(-levels, levels, size=d).astype(np.float32)
            delta = rng.choice([0.0, 1e-7, -1e-7, 1e-6, -1e-6, 3e-5, -3e-5, 1.2e-4, -1.2e-4, 1.3e-4, -1.3e-4, 4e-4],
                               size=d).astype(np.float32)
            x = ((k + np.float32(0.5) + delta) * s).astype(np.float32)
            x = np.clip(x, -amax, amax)
            x[rng.integers(0, d)] = amax * rng.choice([-1.0, 1.0])   # pins the row's absolute maximum
            rows.append(x.astype(np.float32))
    x = np.stack(rows)
    q, s = _quantize_gpu(x, bits)
    with np.errstate(all="ignore"):
        qo, so = orc.quantize_rows(x, bits)
    assert np.array_equal(s.view(np.uint32), so.view(np.uint32))
    assert np.array_equal(q, qo)


def test_quantize_fp16_input():
    rng = np.random.default_rng(3)
    x = rng.standard_normal((300, 128)).astype(np.float16)
    q, s = _quantize_gpu(x, 4)
    qo, so = orc.quantize_rows(x.astype(np.float32), 4)
    assert np.array_equal(q, qo) and np.array_equal(s, so)


def test_quantize_bulk_digest_matches_reference(golden):
    g = golden("quant")
    k, _ = orc.synth_kv(512, 8, 128, seed=3)
    for bits in (2, 3, 4, 8):
        q, s = _quantize_gpu(k, bits)
        sha = lambda a: np.frombuffer(hashlib.sha256(np.ascontiguousarray(a).tobytes()).digest(), dtype=np.uint8)
        assert np.array_equal(sha(q), g[f"quant_bulk_sha_kq{bits}"])
        assert np.array_equal(sha(s), g[f"quant_bulk_sha_ks{bits}"])


@pytest.mark.parametrize("bits", [2, 3, 4, 8])
@pytest.mark.parametrize("n", [1, 3, 8, 17, 100, 1000, 4096 + 5])
def test_pack_unpack_vs_oracle(bits, n):
    L = _lib()
    lo, hi = orc.code_range(bits)
    rng = np.random.default_rng(n + bits)
    codes = rng.integers(lo, hi + 1, size=n).astype(np.int8)
    ct = torch.from_numpy(codes).cuda()
    packed = torch.zeros(orc.packed_size(n, bits), dtype=torch.uint8, device="cuda")
    L.check(L.lib().skv_pack(L.ptr(ct), n, bits, L.ptr(packed), L.stream_ptr()))
    assert np.array_equal(packed.cpu().numpy(), orc.pack_codes(codes, bits))
    back = torch.empty(n, dtype=torch.int8, device="cuda")
    L.check(L.lib().skv_unpack(L.ptr(packed), n, bits, L.ptr(back), L.stream_ptr()))
    assert np.array_equal(back.cpu().numpy(), codes)


def test_pack_empty_and_bad_args():
    L = _lib()
    t = torch.zeros(4, dtype=torch.int8, device="cuda")
    p = torch.zeros(4, dtype=torch.uint8, device="cuda")
    assert L.lib().skv_pack(L.ptr(t), 0, 2, L.ptr(p), L.stream_ptr()) == 0
    assert L.lib().skv_pack(L.ptr(t), 4, 5, L.ptr(p), L.stream_ptr()) < 0
    assert L.lib().skv_pack(None, 4, 2, L.ptr(p), L.stream_ptr()) < 0


@pytest.mark.parametrize("hkv,d", [(4, 64), (8, 128)])
def test_append_then_export_bit_exact(hkv, d):
    from tests.gpu_util import fill_store, make_store, oracle_quantized
    B, n, Lyr = 2, 333, 2
    rng = np.random.default_rng(7)
    bits = rng.choice([2, 3, 4, 8], size=(B, n))
    store = make_store(Lyr, B, hkv, d, hkv * 4, n)
    kv = []
    for layer in range(Lyr):
        ks, vs = zip(*[orc.synth_kv(n, hkv, d, seed=10 * layer + b) for b in range(B)])
        kv.append((np.stack(ks), np.stack(vs)))
    fill_store(store, kv, bits)
    torch.cuda.synchronize()
    assert store.counts.cpu().numpy().tolist() == [[int((bits[b] == w).sum()) for w in (2, 3, 4, 8)] for b in range(B)]
    for layer in range(Lyr):
        for b in range(B):
            ids, wb, kc, vc, ksc, vsc = store.export_sequence(layer, b)
            assert np.array_equal(ids.cpu().numpy(), np.arange(n))
            assert np.array_equal(wb.cpu().numpy(), bits[b])
            kq, vq, kso, vso = oracle_quantized(kv[layer][0][b], kv[layer][1][b], bits[b])
            assert np.array_equal(kc.cpu().numpy(), kq)
            assert np.array_equal(vc.cpu().numpy(), vq)
            assert np.array_equal(ksc.cpu().numpy().view(np.uint32), kso.view(np.uint32))
            assert np.array_equal(vsc.cpu().numpy().view(np.uint32), vso.view(np.uint32))
            # raw packed bytes of every bucket equal the oracle's row packing
            for bi, w in enumerate((2, 3, 4, 8)):
                sel = np.nonzero(bits[b] == w)[0]
                kr, vr, _, _ = store.bucket_rows(layer, b, bi)
                want_k = orc.pack_rows(kq[sel], w).transpose(1, 0, 2)
                want_v = orc.pack_rows(vq[sel], w).transpose(1, 0, 2)
                assert np.array_equal(kr.cpu().numpy(), want_k)
                assert np.array_equal(vr.cpu().numpy(), want_v)


@pytest.mark.parametrize("hkv,d,n,dtype,offset", [
    (1, 64, 37, "f16", 0), (3, 64, 41, "f32", 0), (3, 128, 43, "f16", 0), (1, 128, 5, "f32", 0), (8, 128, 9000, "f16", 0),
    (3, 64, 23001, "f16", 0), (5, 128, 14000, "f32", 0), (4, 64, 50, "f16", 2), (2, 128, 50, "f32", 4)])
def test_bulk_append_rows_of_every_kind(hkv, d, n, dtype, offset):
    """Mixed widths in one call, odd head counts (two tokens meet in one warp at head_dim 64), both numbers of row groups
    per warp and inputs off a 16-byte boundary, with rows of zeros, near-ties, tiny and infinite values: packed bytes
    and scales against the oracle."""
    from tests.gpu_util import make_store, oracle_quantized
    rng = np.random.default_rng(hkv * n + d)
    bits = rng.choice([2, 3, 4, 8], size=(1, n))
    np_t = np.float16 if dtype == "f16" else np.float32
    kv = []
    for i in range(2):
        x = rng.standard_normal((n, hkv, d)).astype(np_t)
        x[0] = 0                                                   # scale 1
        if n > 4:
            lv = np.maximum(2.0 ** (bits[0, 1:4] - 1) - 1, 1)[:, None, None]
            x[1:4] = ((rng.integers(-1, 1, size=(3, hkv, d)) + 0.5) / lv).astype(np_t)   # ties, exact and rounded
            x[1:4, :, 7] = 1.0
            x[4] = (x[4].astype(np.float32) * 1e-7).astype(np_t)   # subnormal halves
            if i == 0:
                x[2, :, 3] = np.inf
        kv.append(x)

    def device(x):
        flat = torch.zeros(x.size + 8, dtype=torch.from_numpy(x).dtype, device="cuda")
        flat[offset:offset + x.size] = torch.from_numpy(x).cuda().view(-1)
        return flat[offset:offset + x.size].view(n, hkv, d)
    store = make_store(1, 1, hkv, d, hkv, n)
    dst = store.plan_bulk(torch.from_numpy(bits.astype(np.int64)).cuda())
    store.append(0, device(kv[0]), device(kv[1]), *dst[:3])
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        kq, vq, ks, vs = oracle_quantized(kv[0].astype(np.float32), kv[1].astype(np.float32), bits[0])
    for bi, w in enumerate((2, 3, 4, 8)):
        sel = np.nonzero(bits[0] == w)[0]
        sel = sel[sel != 2] if n > 4 else sel       # inf / inf has no code the two sides must agree on; its scale is checked
        raw = np.nonzero(bits[0] == w)[0]
        keep = np.isin(raw, sel)
        kr, vr, ksc, vsc = (t.cpu().numpy() for t in store.bucket_rows(0, 0, bi))
        assert np.array_equal(kr[:, keep], orc.pack_rows(kq[sel], w).transpose(1, 0, 2))
        assert np.array_equal(vr[:, keep], orc.pack_rows(vq[sel], w).transpose(1, 0, 2))
        assert np.array_equal(ksc.view(np.uint32), ks[raw].T.view(np.uint32))
        assert np.array_equal(vsc.view(np.uint32), vs[raw].T.view(np.uint32))
