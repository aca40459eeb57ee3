"""Routed experts with f16 activations as rows of MXFP8 pieces against fp64 and against the register-fed f16 kernel."""
import pytest
import torch

from titanic_flash_41_b200.models import engine as E
from titanic_flash_41_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"
PIECES = 6


def _groups(counts, topk):
    """Groups of ``counts`` pairs (expert 2 i + 1 for group i), pairs in shuffled order: the tables of tf_route_group."""
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    n = sum(counts)
    order = torch.randperm(n, generator=torch.Generator().manual_seed(n)).int().to(DEV)
    starts = [sum(counts[:i]) for i in range(len(counts))]
    return i32([2 * i + 1 for i in range(len(counts))]), i32(starts), i32(counts), i32([len(counts)]), order, i32([n])


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("K,I,counts", [(256, 256, [1]), (512, 768, [5, 6, 1]), (768, 256, [24, 3]), (2304, 512, [2, 10, 11]), (1280, 1280, [4])])
def test_split_experts_match_fp64(K, I, counts):
    """Groups of fewer, exactly and more than two rows (passes of the accumulator), inputs ending inside 512, rows of scales on
    and off the 16-byte grain.  Products are exact, so both GEMVs stay within fp32 summation (1e-6); the activation between
    them is rounded to f16 as the register-fed kernel rounds it (2e-3 of the second product's norm covers a last-bit change)."""
    topk, pairs, El = 2, sum(counts), 2 * len(counts) + 1
    T = -(-pairs // topk)
    gen = torch.Generator(device=DEV).manual_seed(K + I)
    x = (torch.randn(T, K, device=DEV, generator=gen) * torch.exp(torch.randn(T, K, device=DEV, generator=gen))).half()
    w1, w3, w2 = (E.quant_mxfp4_device(torch.randn(El, n, k, device=DEV, generator=gen) * 0.05) for n, k in ((I, K), (I, K), (K, I)))
    ge, gs, gc, ng, sp, nl = groups = _groups(counts, topk)
    st, pitch = native.StatusWord(DEV), native.lib().tf_moe_split_pitch
    u8 = lambda *s: torch.full(s, 0x55, dtype=torch.uint8, device=DEV)
    x3, x3s, a3, a3s = u8(PIECES * pairs, K), u8(PIECES * pairs, pitch(K)), u8(PIECES * pairs, I), u8(PIECES * pairs, pitch(I))
    y = torch.full((pairs, K), 7.0, device=DEV)
    native.call("tf_moe_split_rows", x, K, sp, nl, topk, pairs, x3, x3s, K)
    native.call("tf_moe_gemv_split", w1[0], w3[0], w1[1], w3[1], El, x3, x3s, pairs, None, 0, a3, a3s, I, K, ge, gs, gc, ng, sp,
                len(counts), 10.0, st.t)
    native.call("tf_moe_gemv_split", w2[0], None, w2[1], None, El, a3, a3s, pairs, y, K, None, None, K, I, ge, gs, gc, ng, sp,
                len(counts), 0.0, st.t)
    st.check()
    whole = lambda q, s, n: (q.view(torch.float8_e4m3fn).double().view(pairs, PIECES, n // 32, 32)
                             * torch.exp2(s[:, :n // 32].double() - 127).view(pairs, PIECES, n // 32, 1)).sum(1).view(pairs, n)
    rows = x[(sp // topk).long()].double()
    assert torch.equal(whole(x3, x3s, K), rows) and native.lib().tf_moe_split_pieces() == PIECES
    expert = torch.repeat_interleave(ge, gc).long()
    act = whole(a3, a3s, I)                                          # sorted order
    W = [E.dequant_mxfp4(*w).double() for w in (w1, w3, w2)]
    want = torch.empty_like(act)
    for i in range(pairs):
        g, u = (rows[i] @ W[j][expert[i]].t() for j in (0, 1))
        want[i] = torch.nn.functional.silu(g.clamp(max=10.0)) * u.clamp(-10.0, 10.0)
    assert _rel(act, want) < 1e-3                                    # one f16 rounding: 2^-11 at most
    assert _rel(y[sp.long()], torch.stack([act[i] @ W[2][expert[i]].t() for i in range(pairs)])) < 1e-6


def test_split_is_no_less_precise_than_the_register_fed_form():
    """5,120 inputs: the error against fp64 sums of the same f16 inputs (3.8e-8 measured; f16 x f16: 2.3e-7)."""
    K, N, T = 5120, 256, 4
    torch.manual_seed(1)
    pk, sc = E.quant_mxfp4_device(torch.randn(1, N, K, device=DEV) * 0.05)
    x = torch.randn(T, K, device=DEV).half()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    sp, st = torch.arange(T, dtype=torch.int32, device=DEV), native.StatusWord(DEV)
    x3, x3s = torch.zeros(PIECES * T, K, dtype=torch.uint8, device=DEV), torch.zeros(PIECES * T, native.lib().tf_moe_split_pitch(K), dtype=torch.uint8, device=DEV)
    y, f = torch.zeros(T, N, device=DEV), torch.zeros(T, N, device=DEV)
    native.call("tf_moe_split_rows", x, K, sp, i32([T]), 1, T, x3, x3s, K)
    native.call("tf_moe_gemv_split", pk, None, sc, None, 1, x3, x3s, T, y, N, None, None, N, K, i32([0]), i32([0]), i32([T]), i32([1]), sp, 1,
                0.0, st.t)
    native.call("tf_smallm_gemm", 1, pk, None, sc, None, N * (K // 2), N * (K // 32), K // 2, K // 32, x, K, f, N, 0, N, K, 0, i32([0]),
                i32([0]), i32([T]), i32([1]), sp, 1, 1, T, 0.0)
    st.check()
    want = x.double() @ E.dequant_mxfp4(pk, sc)[0].double().t()
    assert _rel(y, want) < 2e-7 and _rel(y, want) <= _rel(f, want)


def test_split_refuses_bad_arguments():
    st, t = native.StatusWord(DEV), torch.zeros(4096, dtype=torch.uint8, device=DEV)
    for N, K in ((128, 256), (256, 128), (256, 384)):               # plain form: N of 256; K of 256
        with pytest.raises(native.NativeError):
            native.call("tf_moe_gemv_split", t, None, t, None, 1, t, t, 1, t, N, None, None, N, K, t, t, t, t, t, 1, 0.0, st.t)


def _both(x, w1, w3, w2, groups, limit):
    """Both GEMVs over the groups: (f16 activations as rows of their pieces' sum, f32 rows by pair)."""
    El, I, K = w1[0].shape[0], w1[0].shape[1], x.shape[1]
    ge, gs, gc, ng, sp, nl = groups
    pairs, pitch, st = sp.numel(), native.lib().tf_moe_split_pitch, native.StatusWord(DEV)
    u8 = lambda *s: torch.full(s, 0x55, dtype=torch.uint8, device=DEV)
    x3, x3s, a3, a3s = u8(PIECES * pairs, K), u8(PIECES * pairs, pitch(K)), u8(PIECES * pairs, I), u8(PIECES * pairs, pitch(I))
    y = torch.full((pairs, K), 7.0, device=DEV)
    native.call("tf_moe_split_rows", x, K, sp, nl, 1, pairs, x3, x3s, K)
    native.call("tf_moe_gemv_split", w1[0], w3[0], w1[1], w3[1], El, x3, x3s, pairs, None, 0, a3, a3s, I, K, ge, gs, gc, ng, sp,
                ge.numel(), limit, st.t)
    native.call("tf_moe_gemv_split", w2[0], None, w2[1], None, El, a3, a3s, pairs, y, K, None, None, K, I, ge, gs, gc, ng, sp,
                ge.numel(), 0.0, st.t)
    st.check()
    return y


@pytest.mark.parametrize("limit", [0.0, 10.0])
def test_rows_that_are_not_finite_stay_so(limit):
    """An infinity or a NaN among a row's inputs, and (without a clamp) a SwiGLU product beyond f16: every output of that row is
    NaN, those of the other rows keep their bits."""
    K = I = 512
    gen = torch.Generator(device=DEV).manual_seed(11)
    x = torch.randn(9, K, device=DEV, generator=gen).half()
    w1, w3, w2 = (E.quant_mxfp4_device(torch.randn(5, n, k, device=DEV, generator=gen) * 0.5) for n, k in ((I, K), (I, K), (K, I)))
    groups = _groups([6, 3], 1)
    clean = _both(x, w1, w3, w2, groups, limit)
    assert bool(torch.isfinite(clean).all())
    bad = x.clone()
    bad[1, 40], bad[2, 77], bad[4, 500] = float("inf"), -float("inf"), float("nan")
    spoilt = [1, 2, 4]
    if limit == 0.0:
        bad[7] *= 200.0                                      # products of 2e5 and more
        spoilt.append(7)
    y = _both(bad, w1, w3, w2, groups, limit)
    kept = [r for r in range(9) if r not in spoilt]
    assert bool(torch.isnan(y[spoilt]).all()) and torch.equal(y[kept], clean[kept])


def test_inputs_of_any_f16_value_are_kept_whole():
    """Blocks of 32 that hold the largest and the smallest f16 numbers at once, and rows whose weights are zero where the large
    ones are: the pieces add up to the inputs exactly, and such a row's sum is as near to fp64 as any (1e-6 covers fp32 summation)."""
    K, N, T = 512, 256, 6
    gen = torch.Generator(device=DEV).manual_seed(12)
    x = torch.randint(-2 ** 15, 2 ** 15, (T, K), dtype=torch.int16, device=DEV, generator=gen).view(torch.float16)
    x = torch.where(torch.isfinite(x), x, torch.full_like(x, 6e-8))
    x[3:, :] = torch.randn(T - 3, K, device=DEV, generator=gen).half() * 0.01
    x[3:, ::32] = 32768.0
    w = torch.randn(1, N, K, device=DEV, generator=gen)
    w[:, :, ::32] = 0.0
    pk, sc = E.quant_mxfp4_device(w)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    sp, st, pitch = torch.arange(T, dtype=torch.int32, device=DEV), native.StatusWord(DEV), native.lib().tf_moe_split_pitch(K)
    x3, x3s = torch.zeros(PIECES * T, K, dtype=torch.uint8, device=DEV), torch.zeros(PIECES * T, pitch, dtype=torch.uint8, device=DEV)
    y = torch.zeros(T, N, device=DEV)
    native.call("tf_moe_split_rows", x, K, sp, i32([T]), 1, T, x3, x3s, K)
    native.call("tf_moe_gemv_split", pk, None, sc, None, 1, x3, x3s, T, y, N, None, None, N, K, i32([0]), i32([0]), i32([T]), i32([1]), sp, 1,
                0.0, st.t)
    st.check()
    pieces = x3.view(torch.float8_e4m3fn).double().view(T, PIECES, K // 32, 32) * torch.exp2(x3s[:, :K // 32].double() - 127).view(T, PIECES, K // 32, 1)
    want = x.double() @ E.dequant_mxfp4(pk, sc)[0].double().t()
    assert _rel(y[3:], want[3:]) < 1e-6
    assert torch.equal(pieces.sum(1).view(T, K), x.double())
