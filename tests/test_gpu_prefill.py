"""The prompt pass (skv_prefill_attention): causal attention over the unquantised prompt and the per-key
attention mass of the importance update, against the oracle's dense fp32 attention with a causal mask
(orc.dequant_attend on codes = values, scale 1) and ImportanceState.update on the resulting probabilities.
Inputs are fp16; the oracle sees the same fp16-rounded numbers.  Tolerance: 2e-3 absolute + 1e-3 relative
on the output (stored as fp16, so one more half-ulp relative), 2e-3 relative on the mass."""
import numpy as np
import pytest
import torch

from oracle import smartkv_oracle as orc
from tests.gpu_util import assert_close

pytestmark = pytest.mark.gpu


def oracle_prefill(q, k, v, group, state):
    """q [n, Hq, D], k / v [n, Hkv, D] fp32 -> (out [n, Hq, D], key mass [n]) for one sequence."""
    n = q.shape[0]
    kk = orc.expand_gqa(k.transpose(1, 0, 2)[None], group)          # [1, Hq, n, D]
    vv = orc.expand_gqa(v.transpose(1, 0, 2)[None], group)
    mask = np.where(np.arange(n)[None, :] > np.arange(n)[:, None], -np.inf, 0.0).astype(np.float32)
    ones = np.ones(kk.shape[:3], np.float32)
    out, probs = orc.dequant_attend(q.transpose(1, 0, 2)[None], kk, ones, vv, ones, mask=mask[None, None])
    mass = state.update(0, probs, list(range(n)))
    return out[0].transpose(1, 0, 2), mass


@pytest.mark.parametrize("hq,hkv,d,n,B", [(32, 4, 64, 200, 2), (32, 8, 128, 131, 1), (8, 8, 64, 64, 1), (16, 2, 128, 1, 1),
                                          (32, 4, 64, 515, 1)])
def test_prefill_attention_and_key_mass(hq, hkv, d, n, B):
    from smartkv_b200.prefill import causal_prefill_attention
    rng = np.random.default_rng(hq + n)
    q = rng.standard_normal((B, n, hq, d)).astype(np.float16)
    k = rng.standard_normal((B, n, hkv, d)).astype(np.float16)
    v = rng.standard_normal((B, n, hkv, d)).astype(np.float16)
    w = rng.uniform(0.5, 1.5, size=(B, hq)).astype(np.float32)
    qt, kt, vt = (torch.from_numpy(x).cuda() for x in (q, k, v))
    out, mass = causal_prefill_attention(qt, kt, vt, torch.from_numpy(w).cuda())
    torch.cuda.synchronize()
    out, mass = out.float().cpu().numpy(), mass.cpu().numpy()
    for b in range(B):
        st = orc.ImportanceState(1)
        # make the oracle's head weights the ones handed to the kernel: the weights are a function of the
        # head EMA, which the oracle updates from the probabilities; fix its output instead
        st.head_weights = lambda probs, wb=w[b]: wb
        ref, ref_mass = oracle_prefill(q[b].astype(np.float32), k[b].astype(np.float32), v[b].astype(np.float32),
                                       hq // hkv, st)
        assert_close(out[b], ref, 2e-3, 2e-3, f"prompt attention, sequence {b}")
        assert np.allclose(mass[b], ref_mass, rtol=2e-3, atol=1e-4), np.abs(mass[b] - ref_mass).max()
        assert abs(mass[b].sum() - n * w[b].sum()) <= 1e-3 * n * w[b].sum()       # every query row sums to one


def test_prefill_accepts_the_transposed_views_of_an_attention_module():
    """q / k / v as a Llama attention holds them: [B, H, n, D] views of [B, n, H*D] projections."""
    from smartkv_b200.prefill import causal_prefill_attention
    B, n, hq, hkv, d = 2, 96, 32, 4, 64
    g = torch.Generator(device="cuda").manual_seed(0)
    qp = torch.randn((B, n, hq * d), generator=g, device="cuda").half()
    kp = torch.randn((B, n, hkv * d), generator=g, device="cuda").half()
    vp = torch.randn((B, n, hkv * d), generator=g, device="cuda").half()
    q, k, v = qp.view(B, n, hq, d), kp.view(B, n, hkv, d), vp.view(B, n, hkv, d)
    out, mass = causal_prefill_attention(q, k, v)
    qh, kh, vh = (x.transpose(1, 2).float() for x in (q, k, v))
    kh, vh = kh.repeat_interleave(hq // hkv, 1), vh.repeat_interleave(hq // hkv, 1)
    s = qh @ kh.transpose(2, 3) / d ** 0.5
    idx = torch.arange(n, device="cuda")
    s = s.masked_fill(idx[None, :] > idx[:, None], float("-inf"))
    p = torch.softmax(s, -1)
    ref = (p @ vh).transpose(1, 2)
    assert torch.allclose(out.float(), ref, atol=2e-3, rtol=2e-3)
    assert torch.allclose(mass, p.sum(dim=(1, 2)), rtol=2e-3, atol=1e-4)


def test_prefill_rejects_what_it_cannot_run():
    from smartkv_b200 import SmartKVLibraryError
    from smartkv_b200.prefill import causal_prefill_attention
    q = torch.randn((1, 8, 4, 64), device="cuda")
    with pytest.raises(TypeError):
        causal_prefill_attention(q, q, q)                                   # fp32
    h = torch.randn((1, 8, 4, 96), device="cuda").half()
    with pytest.raises(SmartKVLibraryError):
        causal_prefill_attention(h, h, h)                                   # head_dim 96


def _dense64(q, k, v, w):
    """fp64 (out [B, n, Hq, D], mass [B, n]) from the same fp16 numbers."""
    B, n, hq, d = q.shape
    qh, kh, vh = (x.transpose(1, 2).double() for x in (q, k, v))
    kh, vh = (x.repeat_interleave(hq // x.shape[1], 1) for x in (kh, vh))
    s = qh @ kh.transpose(2, 3) / d ** 0.5
    s.masked_fill_(torch.ones((n, n), dtype=torch.bool, device=q.device).triu_(1), float("-inf"))
    p = torch.softmax(s, -1)
    return (p @ vh).transpose(1, 2), (p.sum(2) * w.double()[..., None]).sum(1)


# The 128-token tiles: one token short, exact, one over; several tiles; heads in pairs (even groups) and query tiles in
# pairs (odd groups, the second tile missing for an odd number of tiles).  All but two have fewer units than SMs.
@pytest.mark.parametrize("hq,hkv,d,n,B,layout", [
    (4, 2, 128, 127, 1, "token"), (4, 2, 64, 128, 2, "head"), (8, 1, 128, 129, 1, "token"), (3, 1, 64, 256, 1, "token"),
    (3, 3, 128, 257, 2, "head"), (6, 2, 64, 385, 1, "token"), (32, 8, 128, 700, 3, "head"), (32, 4, 64, 1024, 2, "token"),
    (4, 2, 128, 300, 1, "rows"), (4, 2, 64, 300, 2, "expanded"), (4, 1, 64, 40, 1, "grow")])
def test_prefill_tiles_pairs_and_strides(hq, hkv, d, n, B, layout):
    """Against fp64.  Error bounds: P and the output are rounded to fp16 (2^-11 relative each, P's averaging out over the
    keys), so 2e-3 of the result's magnitude leaves a factor of two; the mass is an fp32 sum of at most n * hq terms."""
    from smartkv_b200.prefill import causal_prefill_attention
    g = torch.Generator(device="cuda").manual_seed(n + hq)

    def make(heads):
        if layout == "head":
            return torch.randn((B, heads, n, d), generator=g, device="cuda").half().transpose(1, 2)
        return torch.randn((B, n, heads, d), generator=g, device="cuda").half()
    q, k, v = make(hq), make(hkv), make(hkv)
    if layout == "rows":          # every key token is the same row: stride 0, which no tensor map holds
        k = k[:, :1].expand(B, n, hkv, d)
    elif layout == "expanded":    # one head's and one sequence's data for all of them
        k, v = k[:1, :, :1].expand(B, n, hkv, d), v[:1].expand(B, n, hkv, d)
    elif layout == "grow":        # scores that outgrow the running maximum by far more than 2^8, tile after tile
        n = 500
        q = torch.randn((B, n, hq, d), generator=g, device="cuda").abs().half()
        k = (torch.rand((B, n, hkv, d), generator=g, device="cuda") * torch.linspace(0, 8, n, device="cuda")[:, None, None]).half()
        v = torch.randn((B, n, hkv, d), generator=g, device="cuda").half()
    w = torch.rand((B, hq), generator=g, device="cuda") + 0.5
    out, mass = causal_prefill_attention(q, k, v, w)
    ref, ref_mass = _dense64(q, k, v, w)
    err = (out.double() - ref).abs()
    assert bool((err <= 2e-3 + 2e-3 * ref.abs()).all()), float(err.max())
    assert torch.allclose(mass.double(), ref_mass, rtol=1e-3, atol=1e-5), float((mass.double() - ref_mass).abs().max())
    alone, none = causal_prefill_attention(q, k, v, want_mass=False)
    assert none is None and torch.equal(alone, out)

def _expand64(q, k, v):
    """q, k, v as [B, Hq, n, D] fp64."""
    qh, kh, vh = (x.transpose(1, 2).double() for x in (q, k, v))
    return qh, *(x.repeat_interleave(q.shape[2] // k.shape[2], 1) for x in (kh, vh))


@pytest.mark.parametrize("hq,hkv,d,n,at", [(4, 2, 64, 300, 70), (8, 2, 128, 200, 133), (3, 1, 128, 260, 0), (3, 3, 64, 129, 127)])
@pytest.mark.parametrize("what", ["nan", "no_score"])
def test_prefill_mass_of_keys_a_query_cannot_see(hq, hkv, d, n, at, what):
    """A query whose row is NaN, or that has no finite score, spoils the mass of the keys it sees and of no other; the output of
    every other query stays what it is.  Same bounds as above."""
    from smartkv_b200.prefill import causal_prefill_attention
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn((1, n, h, d), generator=g, device="cuda").half() for h in (hq, hkv, hkv))
    if what == "nan":
        q[0, at, hq - 1] = float("nan")
    else:
        k[..., 0] = -k[..., 0].abs() - 0.5
        q[0, at, hq - 1, 0] = float("inf")           # -inf against every key
    w = torch.rand((1, hq), generator=g, device="cuda") + 0.5
    out, mass = causal_prefill_attention(q, k, v, w)
    qh, kh, vh = _expand64(q, k, v)
    s = (qh @ kh.transpose(2, 3) / d ** 0.5).masked_fill_(torch.ones((n, n), dtype=torch.bool, device="cuda").triu_(1), float("-inf"))
    p = torch.softmax(s, -1)
    ref = (p @ vh).transpose(1, 2)
    p[:, hq - 1, at] = 0
    ref_mass = (p.sum(2) * w.double()[..., None]).sum(1)
    assert torch.allclose(mass[:, at + 1:].double(), ref_mass[:, at + 1:], rtol=1e-3, atol=1e-5), mass[:, at + 1:]
    assert not bool(mass[:, :at + 1].isfinite().any())
    others = torch.ones((n, hq), dtype=torch.bool, device="cuda")
    others[at, hq - 1] = False
    err = (out[0].double() - ref[0]).abs()[others]
    assert bool((err <= 2e-3 + 2e-3 * ref[0].abs()[others]).all())


@pytest.mark.parametrize("hq,hkv,d,n,at", [(4, 2, 64, 300, 112), (8, 2, 128, 256, 255), (3, 1, 128, 260, 16), (2, 2, 64, 140, 129)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_prefill_output_of_queries_before_a_non_finite_value_row(hq, hkv, d, n, at, value):
    """A value row that is not finite reaches the queries that see it, and of the ones before it at most those of its own group
    of 16 positions (their weight for it is zero, and zero times infinity is not).  Same bounds as above."""
    from smartkv_b200.prefill import causal_prefill_attention
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn((1, n, h, d), generator=g, device="cuda").half() for h in (hq, hkv, hkv))
    v[0, at, hkv - 1] = value
    out, _ = causal_prefill_attention(q, k, v, want_mass=False)
    first = at // 16 * 16
    ref, _ = _dense64(q[:, :first], k[:, :first], v[:, :first], torch.ones((1, hq), device="cuda"))
    err = (out[:, :first].double() - ref).abs()
    assert bool((err <= 2e-3 + 2e-3 * ref.abs()).all())
    assert not bool(out[0, at:, hq - 1].isfinite().any())
    if hkv > 1:
        assert bool(out[0, :, 0].isfinite().all())


@pytest.mark.parametrize("hq,hkv,d,n,B", [(4, 2, 128, 700, 2), (3, 1, 64, 520, 1)])
def test_prefill_log_sum_exp_at_large_logits(hq, hkv, d, n, B):
    """The row normalisers against 64 bits.  Queries and keys are small whole numbers, so that the scores, in the thousands, are
    exact in fp32; what is left is the rounding of the result, half a unit in its last place, and 2^-21 for the exponentials
    and the sum.  A normaliser that does not belong to the maximum the sum was taken against is off by up to another half unit."""
    import ctypes
    from smartkv_b200 import _lib
    from smartkv_b200.prefill import _strides
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k = (torch.randint(-24, 25, (B, n, h, d), generator=g, device="cuda").half() for h in (hq, hkv))
    k *= torch.linspace(0.25, 1, n, device="cuda").mul(4).round().div(4).half()[None, :, None, None]      # maxima that grow
    v = torch.zeros_like(k)
    out, lse = torch.empty_like(q), torch.empty((B, hq, n), device="cuda")
    _lib.check(_lib.lib().skv_prefill_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), _lib.DTYPE_F16, B, n, hq, hkv, d, _strides(q),
                                                _strides(k), _strides(v), None, out.data_ptr(), lse.data_ptr(), None,
                                                torch.cuda.current_stream().cuda_stream))
    qh, kh, _ = _expand64(q, k, v)
    scale = np.float32(1.4426950408889634) / np.sqrt(np.float32(d))
    s = qh @ kh.transpose(2, 3) * float(scale)
    s.masked_fill_(torch.ones((n, n), dtype=torch.bool, device="cuda").triu_(1), float("-inf"))
    m = s.max(-1, keepdim=True).values
    ref = (m + torch.log2(torch.exp2(s - m).sum(-1, keepdim=True)))[..., 0]
    ulp = torch.exp2(torch.floor(torch.log2(ref.abs().clamp(min=1e-3))) - 23)
    assert float(ref.abs().max()) > 256
    worst = ((lse.double() - ref).abs() - 2.0 ** -21) / ulp
    assert float(worst.max()) <= 0.5, float(worst.max())


@pytest.mark.parametrize("hq,hkv,d,n,B,layout", [(32, 8, 128, 700, 3, "token"), (3, 1, 64, 385, 2, "token"), (4, 2, 128, 300, 1, "rows")])
def test_prefill_wait_that_runs_out_sets_the_error_flag(hq, hkv, d, n, B, layout):
    """With the limit below one poll every role gives up on the first thing that is not ready yet: the launches return, the flag
    is 1, what was owed is NaN, and the very next call in the stream, on the same shared and tensor memory, is right again."""
    import ctypes
    from smartkv_b200 import _lib
    from smartkv_b200.prefill import causal_prefill_attention
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v = (torch.randn((B, n, h, d), generator=g, device="cuda").half() for h in (hq, hkv, hkv))
    if layout == "rows":
        k = k[:, :1].expand(B, n, hkv, d)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    good = causal_prefill_attention(q, k, v, error_flag=err)
    assert int(err) == 0
    lib, value = _lib.lib(), ctypes.c_int32(0)
    try:
        assert lib.skv_set_wait_limit(1) == 0
        out, mass = causal_prefill_attention(q, k, v, error_flag=err)
        plain, _ = causal_prefill_attention(q, k, v)
    finally:
        assert lib.skv_set_wait_limit(1 << 24) == 0
    again = causal_prefill_attention(q, k, v)
    rc = lib.skv_read_error_flag(err.data_ptr(), ctypes.byref(value), torch.cuda.current_stream().cuda_stream)
    assert value.value == 1 and b"timed out" in lib.skv_status_string(rc)
    assert bool(out.isnan().any()) and bool(mass.isnan().any()) and bool(plain.isnan().any())
    assert torch.equal(again[0], good[0]) and torch.equal(again[1], good[1])
    with pytest.raises(ValueError):
        causal_prefill_attention(q, k, v, error_flag=torch.zeros(1, dtype=torch.int32))


def _check64(q, k, v, w):
    """Against fp64, the bounds of test_prefill_tiles_pairs_and_strides."""
    from smartkv_b200.prefill import causal_prefill_attention
    out, mass = causal_prefill_attention(q, k, v, w)
    ref, ref_mass = _dense64(q, k, v, w)
    err = (out.double() - ref).abs()
    assert bool((err <= 2e-3 + 2e-3 * ref.abs()).all()), float(err.max())
    assert torch.allclose(mass.double(), ref_mass, rtol=1e-3, atol=1e-5), float((mass.double() - ref_mass).abs().max())


# On 148 SMs: three to six units a CTA in pass 1 and two to six in pass 2, which carry barrier phases, accumulators and buffers from
# one unit to the next; even groups, odd groups whose second query tile is missing in every other unit, one head per group.
@pytest.mark.parametrize("hq,hkv,d,n,B", [(32, 8, 128, 700, 10), (32, 4, 64, 515, 24), (12, 4, 64, 300, 24), (9, 9, 128, 257, 30),
                                          (24, 8, 128, 385, 16)])
def test_prefill_many_units_a_cta(hq, hkv, d, n, B):
    g = torch.Generator(device="cuda").manual_seed(n + hq)
    q, k, v = (torch.randn((B, n, h, d), generator=g, device="cuda").half() for h in (hq, hkv, hkv))
    _check64(q, k, v, torch.rand((B, hq), generator=g, device="cuda") + 0.5)


@pytest.mark.parametrize("hq,hkv,d,n,B", [(4, 2, 128, 300, 1), (3, 1, 64, 260, 2), (5, 5, 128, 140, 40)])
@pytest.mark.parametrize("rows", ["q", "v", "qk", "kv", "qkv"])
def test_prefill_tensors_copied_row_by_row(hq, hkv, d, n, B, rows):
    """Every token of the named tensors is the same row: stride 0, which no tensor map holds, so the loading warp copies the tiles."""
    g = torch.Generator(device="cuda").manual_seed(n + d)
    make = lambda name, h: (torch.randn((B, 1 if name in rows else n, h, d), generator=g, device="cuda").half().expand(B, n, h, d))
    _check64(make("q", hq), make("k", hkv), make("v", hkv), torch.rand((B, hq), generator=g, device="cuda") + 0.5)
