"""Numerics of the CUDA kernels against plain PyTorch fp32 references (one B200)."""
import math

import numpy as np
import pytest
import torch

from titanic_flash_41_b200.formats import codecs
from titanic_flash_41_b200.models import engine as E
from titanic_flash_41_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return float((a.float() - b.float()).norm() / (b.float().norm() + 1e-12))


@pytest.mark.parametrize("M", [1, 5, 8, 16, 27, 32])
def test_smallm_fp8_dense(M):
    torch.manual_seed(M)
    N, K = 384, 1024
    w = torch.randn(N, K, device=DEV) * 0.05
    fw = E.quant_fp8_device(w)
    x = torch.randn(M, K, device=DEV).half()
    out = torch.zeros(M, N, device=DEV)
    native.call("tf_smallm_gemm", 0, fw.q, None, fw.s, None, 0, 0, K, K // 128, x, K, out, N, 0, N, K, M,
                None, None, None, None, None, 1, 0, M, 0.0)
    ref = x.float() @ E.dequant_fp8(fw).t()
    assert _rel(out, ref) < 2e-3


@pytest.mark.parametrize("M,N,K", [(16, 256, 2048), (9, 384, 4096), (16, 128, 2176)])
def test_smallm_fp8_dense_eight_way_k_split(M, N, K):
    """Dense matrices with few 32-feature tiles and long rows split K over eight warps per CTA
    (K not a multiple of 8 x 128 leaves the last warps short or idle); results are run-to-run identical."""
    torch.manual_seed(K + M)
    fw = E.quant_fp8_device(torch.randn(N, K, device=DEV) * 0.05)
    x = torch.randn(M, K, device=DEV).half()
    outs = []
    for _ in range(2):
        out = torch.zeros(M, N, device=DEV)
        native.call("tf_smallm_gemm", 0, fw.q, None, fw.s, None, 0, 0, K, K // 128, x, K, out, N, 0, N, K, M,
                    None, None, None, None, None, 1, 0, M, 0.0)
        outs.append(out)
    ref = x.float() @ E.dequant_fp8(fw).t()
    assert _rel(outs[0], ref) < 2e-3
    assert torch.equal(outs[0], outs[1])


def test_smallm_fp8_dual_swiglu_and_kslice():
    torch.manual_seed(0)
    N, K, M = 256, 512, 7
    w1, w3 = (E.quant_fp8_device(torch.randn(N, K, device=DEV) * 0.1) for _ in range(2))
    x = torch.randn(M, K, device=DEV).half()
    out = torch.zeros(M, N, device=DEV, dtype=torch.float16)
    native.call("tf_smallm_gemm", 0, w1.q, w3.q, w1.s, w3.s, 0, 0, K, K // 128, x, K, out, N, 1, N, K, M,
                None, None, None, None, None, 1, 0, M, 10.0)
    g = torch.clamp(x.float() @ E.dequant_fp8(w1).t(), max=10.0)
    u = torch.clamp(x.float() @ E.dequant_fp8(w3).t(), -10.0, 10.0)
    assert _rel(out, g * torch.sigmoid(g) * u) < 3e-3


@pytest.mark.parametrize("M,N,K,kind", [(1, 128, 128, "fp8"), (8, 384, 1152, "fp8"), (17, 384, 1280, "fp8"), (24, 12800, 384, "fp8"),
                                        (32, 256, 2176, "fp8"), (9, 12800, 256, "dual"), (25, 256, 1152, "dual"), (3, 128, 128, "dual"),
                                        (4, 12800, 128, "bf16"), (24, 256, 640, "bf16"), (32, 128, 1152, "bf16")])
def test_smallm_dense_stream(M, N, K, kind):
    """One to four 8-row tiles with ragged last ones; fewer K blocks than warps, one or two blocks more than a
    multiple of eight, and more feature tiles than resident CTAs (the copies then run across tiles).

    Against fp64 of the same stored values: products are exact in fp32, sums of K terms in fp32."""
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16 if kind == "bf16" else torch.float16)
    out = torch.full((M + 1, N), 9.0, device=DEV)
    if kind == "bf16":
        w = (torch.randn(N, K, device=DEV) * 0.05).bfloat16()
        native.call("tf_smallm_gemm", 2, w, None, None, None, 0, 0, K * 2, 0, x, K, out, N, 0, N, K, M,
                    None, None, None, None, None, 1, 0, M, 0.0)
        want = x.double() @ w.double().t()
    else:
        ws = [E.quant_fp8_device(torch.randn(N, K, device=DEV) * 0.05 * (1 + torch.arange(N, device=DEV)[:, None] // 128))
              for _ in range(2 if kind == "dual" else 1)]
        w3 = ws[1] if kind == "dual" else None
        native.call("tf_smallm_gemm", 0, ws[0].q, w3.q if w3 else None, ws[0].s, w3.s if w3 else None, 0, 0, K, K // 128,
                    x, K, out, N, 0, N, K, M, None, None, None, None, None, 1, 0, M, 4.0)
        want = x.double() @ E.dequant_fp8(ws[0]).double().t()
        if w3 is not None:
            want = want.clamp(max=4.0)
            want = want * torch.sigmoid(want) * (x.double() @ E.dequant_fp8(w3).double().t()).clamp(-4.0, 4.0)
    assert float((out[:M].double() - want).norm() / want.norm()) < 2e-6 * K ** 0.5
    assert (out[M] == 9.0).all()


@pytest.mark.parametrize("M,kind,okind", [(33, "fp8", 1), (70, "dual", 0), (64, "bf16", 2), (96, "fp8", 0)])
def test_smallm_dense_of_more_rows_than_a_pass(M, kind, okind):
    """Ungrouped matrices with more than 32 rows go through the dense form 32 rows at a time: ragged and full last passes, a
    padded output pitch and the three output types.  fp32 sums of K exact products, then one rounding of the output type."""
    torch.manual_seed(M)
    N, K = 256, 1152
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16 if kind == "bf16" else torch.float16)
    out = torch.full((M + 1, N + 8), 9.0, device=DEV, dtype=(torch.float32, torch.float16, torch.bfloat16)[okind])
    ws = [E.quant_fp8_device(torch.randn(N, K, device=DEV) * 0.05) for _ in range(2)]
    wb = (torch.randn(N, K, device=DEV) * 0.05).bfloat16()
    if kind == "bf16":
        native.call("tf_smallm_gemm", 2, wb, None, None, None, 0, 0, K * 2, 0, x, K, out, N + 8, okind, N, K, M,
                    None, None, None, None, None, 1, 0, M, 0.0)
        want = x.double() @ wb.double().t()
    else:
        w3 = ws[1] if kind == "dual" else None
        native.call("tf_smallm_gemm", 0, ws[0].q, w3.q if w3 else None, ws[0].s, w3.s if w3 else None, 0, 0, K, K // 128,
                    x, K, out, N + 8, okind, N, K, M, None, None, None, None, None, 1, 0, M, 0.0)
        want = x.double() @ E.dequant_fp8(ws[0]).double().t()
        if w3 is not None:
            want = want * torch.sigmoid(want) * (x.double() @ E.dequant_fp8(w3).double().t())
    err = float((out[:M, :N].double() - want).norm() / want.norm())
    assert err < 2e-6 * K ** 0.5 + (0.0, 2.0 ** -11, 2.0 ** -8)[okind]
    assert (out[M] == 9.0).all() and (out[:, N:] == 9.0).all()


def test_smallm_bf16_head():
    torch.manual_seed(1)
    N, K, M = 2048, 512, 9
    w = (torch.randn(N, K, device=DEV) * 0.05).bfloat16()
    x = torch.randn(M, K, device=DEV).bfloat16()
    out = torch.zeros(M, N, device=DEV)
    native.call("tf_smallm_gemm", 2, w, None, None, None, 0, 0, K * 2, 0, x, K, out, N, 0, N, K, M,
                None, None, None, None, None, 1, 0, M, 0.0)
    assert _rel(out, x.float() @ w.float().t()) < 1e-3


def _group_tables(ids, e_lo, e_hi):
    T, k = ids.shape
    i32 = dict(dtype=torch.int32, device=DEV)
    El = e_hi - e_lo
    t = dict(ge=torch.zeros(El, **i32), gs=torch.zeros(El, **i32), gc=torch.zeros(El, **i32),
             ng=torch.zeros(1, **i32), sp=torch.zeros(T * k, **i32), nl=torch.zeros(1, **i32))
    native.call("tf_route_group", ids, T * k, e_lo, e_hi, t["ge"], t["gs"], t["gc"], t["ng"], t["sp"], t["nl"])
    return t


def test_grouped_mxfp4_experts():
    torch.manual_seed(2)
    El, I, d, T, k = 6, 256, 512, 11, 2
    w1, w3 = torch.randn(El, I, d, device=DEV) * 0.05, torch.randn(El, I, d, device=DEV) * 0.05
    w2 = torch.randn(El, d, I, device=DEV) * 0.05
    (p1, s1), (p3, s3), (p2, s2) = (E.quant_mxfp4_device(w) for w in (w1, w3, w2))
    ids = torch.stack([torch.randperm(8, device=DEV)[:k] for _ in range(T)]).int()   # experts 0..7, local 1..6
    e_lo, e_hi = 1, 7
    t = _group_tables(ids, e_lo, e_hi)
    h = torch.randn(T, d, device=DEV).half()
    act = torch.zeros(T * k, I, device=DEV, dtype=torch.float16)
    y = torch.zeros(T * k, d, device=DEV)
    native.call("tf_smallm_gemm", 1, p1, p3, s1, s3, I * d // 2, I * d // 32, d // 2, d // 32, h, d, act, I,
                1, I, d, 0, t["ge"], t["gs"], t["gc"], t["ng"], t["sp"], k, El, 16, 10.0)
    native.call("tf_smallm_gemm", 1, p2, None, s2, None, d * I // 2, d * I // 32, I // 2, I // 32, act, I, y, d,
                0, d, I, 0, t["ge"], t["gs"], t["gc"], t["ng"], t["sp"], 1, El, 16, 0.0)
    d1, d3, d2 = E.dequant_mxfp4(p1, s1), E.dequant_mxfp4(p3, s3), E.dequant_mxfp4(p2, s2)
    for r in range(T):
        for j in range(k):
            e = int(ids[r, j]) - e_lo
            if not 0 <= e < El:
                continue
            g = torch.clamp(h[r].float() @ d1[e].t(), max=10.0)
            u = torch.clamp(h[r].float() @ d3[e].t(), -10.0, 10.0)
            a = (g * torch.sigmoid(g) * u)
            assert _rel(act[r * k + j], a) < 5e-3
            assert _rel(y[r * k + j], act[r * k + j].float() @ d2[e].t()) < 5e-3


def test_add_norm_and_fp8_quant():
    torch.manual_seed(3)
    T, d = 5, 512
    x = torch.randn(T, d, device=DEV).bfloat16()
    delta = torch.randn(T, d, device=DEV)
    w = (1 + 0.1 * torch.randn(d, device=DEV)).bfloat16()
    x0 = x.clone()
    h16 = torch.zeros(T, d, device=DEV, dtype=torch.float16)
    q8 = torch.zeros(T, d, device=DEV, dtype=torch.uint8)
    qs = torch.zeros(T, d // 128, device=DEV)
    native.call("tf_add_norm", x, delta, 0, d, w, h16, None, q8, qs, T, d, 1e-6)
    xr = (x0.float() + delta).bfloat16().float()
    assert torch.equal(x.float(), xr)
    ref = (xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-6) * w.float())
    assert _rel(h16, ref) < 5e-3
    deq = q8.view(torch.float8_e4m3fn).float().view(T, d // 128, 128) * qs[:, :, None]
    assert _rel(deq.view(T, d), ref) < 4e-2


def test_router_matches_oracle():
    from titanic_flash_41_b200.config import tiny_config
    from titanic_flash_41_b200.models.oracle import route
    torch.manual_seed(4)
    T, Ex, d, k = 13, 64, 512, 6
    cfg = tiny_config(n_experts=Ex, topk=k, scoring="sqrtsoftplus", router_bias=True, route_scale=1.5)
    h = torch.randn(T, d, device=DEV).half()
    gate = (torch.randn(Ex, d, device=DEV) / math.sqrt(d)).bfloat16()
    bias = torch.randn(Ex, device=DEV) * 0.1
    logits = torch.zeros(T, Ex, device=DEV)
    ids = torch.zeros(T, k, device=DEV, dtype=torch.int32)
    wts = torch.zeros(T, k, device=DEV)
    native.call("tf_router", h, gate, bias, None, None, -1, logits, ids, wts, T, Ex, d, k, 1, 1, 1.5)
    ref_logits = h.float() @ gate.float().t()
    assert _rel(logits, ref_logits) < 1e-4
    rid, rw = route(logits.cpu(), cfg, bias.cpu())
    assert torch.equal(ids.cpu().long(), rid)
    assert torch.allclose(wts.cpu(), rw, atol=1e-5)


@pytest.mark.parametrize("Hi", [4, 8, 16, 32])
def test_index_scores_and_topk(Hi):
    torch.manual_seed(5)
    T, Di, C, k = 8, 128, 700, 64
    keys_f = torch.randn(2, C, Di)
    krow = Di // 2 + Di // 32
    enc = codecs.index_key_encode(keys_f)                          # [2, C, 68]
    kd = codecs.index_key_decode(enc, Di)
    keys = enc.to(DEV).contiguous()
    q = torch.randn(T, Hi, Di, device=DEV).bfloat16()
    w = torch.rand(T, Hi, device=DEV)
    region = torch.tensor([0] * 4 + [1] * 4, dtype=torch.int32, device=DEV)
    nvalid = torch.tensor([700, 650, 3, 0, 129, 128, 127, 64], dtype=torch.int32, device=DEV)
    scores = torch.full((T, 1024), 7.0, device=DEV)
    native.call("tf_index_scores", q, w, region, nvalid, keys, C * krow, krow, T, Hi, Di, 4, scores, 1024, 0, 700)
    ref = torch.einsum("thd,tcd->thc", q.float().cpu(), kd[region.cpu().long()]).relu()
    ref = (ref * w.cpu()[:, :, None]).sum(1)
    for r in range(T):
        n = int(nvalid[r])
        assert torch.allclose(scores[r, :n].cpu(), ref[r, :n], atol=2e-2, rtol=2e-3)
    sel = torch.zeros(T, k, dtype=torch.int32, device=DEV)
    cnt = torch.zeros(T, dtype=torch.int32, device=DEV)
    # duplicate values to exercise ties
    scores[0, 10:20] = scores[0, 5].item()
    native.call("tf_topk_select", scores, 1024, nvalid, k, sel, cnt, None, 0, T)
    for r in range(T):
        n = int(nvalid[r])
        s = scores[r, :n].cpu()
        got = sel[r].cpu().tolist()
        if n <= k:
            assert got == list(range(n)) + [-1] * (k - n) and int(cnt[r]) == n
            continue
        order = torch.sort(s, descending=True, stable=True).indices[:k]
        assert got == sorted(order.tolist())


@pytest.mark.parametrize("Dh,Hl", [(128, 4), (512, 4), (512, 20), (256, 16)])
def test_sparse_attention_matches_reference(Dh, Hl):
    """Dh 128 runs the register-resident kernel, 256 / 512 the wide-latent one (head dim split over warps)."""
    torch.manual_seed(6)
    T, window, ring, C, k = 6, 16, 64, 50, 12
    win_row, comp_row = -(-(Dh + Dh // 32) // 16) * 16, -(-(Dh // 2 + Dh // 16) // 16) * 16
    kv = torch.randn(2, ring, Dh) * 1.5
    win = torch.zeros(2, ring, win_row, dtype=torch.uint8)
    win[:, :, :Dh + Dh // 32] = codecs.kv_v41_encode(kv)
    kvd = codecs.kv_v41_decode(win, Dh)
    ck = torch.randn(2, C, Dh)
    comp = torch.zeros(2, C, comp_row, dtype=torch.uint8)
    comp[:, :, :Dh // 2 + Dh // 16] = codecs.kv_v41fp4_encode(ck)
    ckd = codecs.kv_v41fp4_decode(comp, Dh)
    pos = torch.tensor([3, 20, 70, 100, 5, 64], dtype=torch.int32)
    region = torch.tensor([0, 0, 0, 1, 1, 1], dtype=torch.int32)
    sel = torch.full((T, k), -1, dtype=torch.int32)
    for r in range(T):
        n = [0, 3, 12, 12, 1, 7][r]
        sel[r, :n] = torch.sort(torch.randperm(C)[:n]).values.int()
    q = (torch.randn(T, Hl, Dh) * 0.5).bfloat16()
    sink = torch.randn(Hl) * 0.5
    freqs = torch.tensor([10000.0 ** (-2.0 * j / 64) for j in range(32)])
    nsplit = 3
    dev = lambda t: t.to(DEV).contiguous()
    part_o = torch.zeros(T, nsplit, Hl, Dh, device=DEV)
    part_lse = torch.zeros(T, nsplit, Hl, device=DEV)
    out = torch.zeros(T, Hl * Dh, device=DEV, dtype=torch.float16)
    st = native.StatusWord(DEV)
    native.call("tf_sparse_attention", dev(q), T, Hl, Dh, dev(pos), dev(region), None, dev(win), ring * win_row,
                win_row, ring, window, dev(comp), C * comp_row, comp_row, dev(sel), k, None, C,
                1 / math.sqrt(Dh), nsplit, part_o, part_lse, dev(sink), dev(freqs), 64, out, None, Hl * Dh, st.t)
    st.check()
    from titanic_flash_41_b200.models.oracle import apply_rope
    for r in range(T):
        p, rg = int(pos[r]), int(region[r])
        nw = min(p + 1, window)
        ks = [kvd[rg, (p - nw + 1 + i) % ring] for i in range(nw)]
        ks += [ckd[rg, int(c)] for c in sel[r] if c >= 0]
        Kmat = torch.stack(ks)
        lg = q[r].float() @ Kmat.t() / math.sqrt(Dh)
        lg = torch.cat([lg, sink[:, None]], 1)
        P = torch.softmax(lg, -1)[:, :-1]
        o = apply_rope((P @ Kmat)[None], torch.tensor([p]), freqs, inverse=True)[0]
        assert _rel(out[r].cpu().view(Hl, Dh), o) < 1e-2, r


@pytest.mark.parametrize("Hl", [64, 20])
def test_sparse_attention_of_prefill_rows_on_tcgen05_matches_reference(Hl):
    """64 rows or more of one split (head dim 128) run on the tcgen05 kernel (heads as M, 128-key
    chunks, S / O in tensor memory): same result as the fp32 reference and as the mma.sync kernel,
    for short rows (window only), rows with several chunks and a partly filled last chunk."""
    torch.manual_seed(8 + Hl)
    T, Dh, window, ring, C, k = 200, 128, 128, 512, 700, 320
    win_row, comp_row = -(-(Dh + Dh // 32) // 16) * 16, -(-(Dh // 2 + Dh // 16) // 16) * 16
    kv = torch.randn(2, ring, Dh) * 1.5
    win = torch.zeros(2, ring, win_row, dtype=torch.uint8)
    win[:, :, :Dh + Dh // 32] = codecs.kv_v41_encode(kv)
    kvd = codecs.kv_v41_decode(win, Dh)
    ck = torch.randn(2, C, Dh)
    comp = torch.zeros(2, C, comp_row, dtype=torch.uint8)
    comp[:, :, :Dh // 2 + Dh // 16] = codecs.kv_v41fp4_encode(ck)
    ckd = codecs.kv_v41fp4_decode(comp, Dh)
    pos = torch.cat([torch.arange(0, 100), torch.arange(300, 400)]).int()            # short windows, then full ones
    region = torch.cat([torch.zeros(100), torch.ones(100)]).int()
    sel = torch.full((T, k), -1, dtype=torch.int32)
    cnt = torch.zeros(T, dtype=torch.int32)
    for r in range(T):
        n = [0, 1, 37, 128, 129, 255, 320][r % 7]
        sel[r, :n] = torch.sort(torch.randperm(C)[:n]).values.int()
        cnt[r] = n
    q = (torch.randn(T, Hl, Dh) * 0.5).bfloat16()
    sink = torch.randn(Hl) * 0.5
    freqs = torch.tensor([10000.0 ** (-2.0 * j / 64) for j in range(32)])
    dev = lambda t: t.to(DEV).contiguous()
    st = native.StatusWord(DEV)
    outs = []
    for tc_on, counts in ((1, None), (1, dev(cnt)), (0, None)):
        native.lib().tf_sparse_attention_set_tc(tc_on)
        part_o = torch.zeros(T, 1, Hl, Dh, device=DEV)
        part_lse = torch.zeros(T, 1, Hl, device=DEV)
        out = torch.zeros(T, Hl * Dh, device=DEV, dtype=torch.float16)
        try:
            native.call("tf_sparse_attention", dev(q), T, Hl, Dh, dev(pos), dev(region), None, dev(win), ring * win_row,
                        win_row, ring, window, dev(comp), C * comp_row, comp_row, dev(sel), k, counts, C,
                        1 / math.sqrt(Dh), 1, part_o, part_lse, dev(sink), dev(freqs), 64, out, None, Hl * Dh, st.t)
            torch.cuda.synchronize()
        finally:
            native.lib().tf_sparse_attention_set_tc(1)
        st.check()
        outs.append(out.cpu().view(T, Hl, Dh).float())
    from titanic_flash_41_b200.models.oracle import apply_rope
    worst = 0.0
    for r in range(T):
        p, rg = int(pos[r]), int(region[r])
        nw = min(p + 1, window)
        ks = [kvd[rg, (p - nw + 1 + i) % ring] for i in range(nw)]
        ks += [ckd[rg, int(c)] for c in sel[r] if c >= 0]
        Kmat = torch.stack(ks)
        lg = q[r].float() @ Kmat.t() / math.sqrt(Dh)
        lg = torch.cat([lg, sink[:, None]], 1)
        P = torch.softmax(lg, -1)[:, :-1]
        o = apply_rope((P @ Kmat)[None], torch.tensor([p]), freqs, inverse=True)[0]
        for got in outs:
            worst = max(worst, _rel(got[r], o))
    assert worst < 1.5e-2, worst
    assert _rel(outs[0], outs[2]) < 1e-2 and torch.equal(outs[0], outs[1])


def test_softmax_sum_of_a_long_row_does_not_gather_rounding():
    """Prefill rows of 8,192 keys whose probabilities are 0.75 and a little (not an f16 number, its f16 copy is 0.75), so that
    every addition to the running sum rounds the same way: the products with the values are exact, what is left is the error of
    the sum.  In one chain over the row it is 1.4e-5 on average (emulated in fp32), closed at every chunk 4.3e-7 (9.2e-7 at most).
    A half-ulp of f16 is 2.4e-4 to 4.9e-4, the sinks spread the rows over it evenly: a relative error of r turns one output in
    5e-4 / r to its neighbour: 2.7 % of them against 0.1 %."""
    torch.manual_seed(2)
    T, Hl, Dh, k, C = 64, 64, 128, 8192, 2
    d = (torch.rand(T, Hl, dtype=torch.float64) * 2 - 1) * 0.9 * 2.0 ** -12
    x = torch.log2(0.75 + d)
    q = torch.zeros(T, Hl, Dh)
    left = (x * 2.0 ** 22).round() * 2.0 ** -22              # as three bf16 numbers
    for i in range(3):
        q[:, :, i] = left.bfloat16().float()
        left = left - q[:, :, i].double()
    assert bool((left == 0).all())
    comp = torch.zeros(1, C, 80, dtype=torch.uint8)          # 64 bytes of e2m1 pairs, eight e4m3 scales
    code = torch.randint(1, 8, (Dh,))
    code[:16] = 0
    scale = torch.randint(0x38, 0x40, (8,))
    for j in range(C):                                       # key 1 meets the three parts of q, key 0 does not
        c = code.clone()
        c[:3] = 2 * j
        comp[0, j, :64] = (c[0::2] | c[1::2] << 4).to(torch.uint8)
        comp[0, j, 64:72] = scale.to(torch.uint8)
    comp[:, :, 64] = 0x38
    value = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64)[code] * (1 + (scale - 0x38) / 8.0).repeat_interleave(16).double()
    sel = torch.ones(T, k, dtype=torch.int32)
    sel[:, 0] = sel[:, 64] = 0                               # the reference maximum of both halves: score 0
    total = 2 + (k - 2) * (0.75 + d)
    sink = torch.log(torch.rand(Hl) * 2e-3 * float(total.mean()) + 1e-3)
    pos = torch.arange(T, dtype=torch.int32) + 300
    dev = lambda t: t.to(DEV).contiguous()
    st, out = native.StatusWord(DEV), torch.zeros(T, Hl * Dh, device=DEV, dtype=torch.float16)
    part, lse = torch.zeros(T, 1, Hl, Dh, device=DEV), torch.zeros(T, 1, Hl, device=DEV)
    win = torch.zeros(1, 512, 144, dtype=torch.uint8, device=DEV)
    native.call("tf_sparse_attention", dev(q.bfloat16()), T, Hl, Dh, dev(pos), dev(torch.zeros(T, dtype=torch.int32)), dev(pos + 1), win,
                512 * 144, 144, 512, 128, dev(comp), C * 80, 80, dev(sel), k, dev(torch.full((T,), k, dtype=torch.int32)), C,
                math.log(2.0), 1, part, lse, dev(sink), torch.zeros(32, device=DEV), 64, out, None, Hl * Dh, st.t)
    st.check()
    weight = (2 + (k - 2) * 0.75) / (total + sink.double().exp())
    want = (weight[:, :, None] * value[16:]).half()
    moved = float((out.cpu().view(T, Hl, Dh)[:, :, 16:] != want).float().mean())
    assert moved < 5e-3, moved


@pytest.mark.parametrize("Dh", [128, 512])
@pytest.mark.parametrize("Hl,drift", [(64, 0.0), (64, 12.0), (33, 12.0), (1, 0.0)])
def test_sparse_attention_of_more_rows_than_ctas_and_moving_maximum(Hl, drift, Dh):
    """Three to seven query rows a CTA (two CTAs an SM at head dim 128, one at 512) with one to seven chunks each, rows without
    any key among them, so that every barrier passes from row to row in both phases, and head counts that leave a softmax warp idle; ``drift`` makes later keys' scores grow by
    hundreds, so that the reference maximum moves in some heads at every chunk and O and the sum are rescaled.

    P is f16 (2^-11 relative), keys are exact in f16, the output is f16: within 1e-3 of fp64."""
    from titanic_flash_41_b200.models.oracle import apply_rope
    torch.manual_seed(31 + Hl)
    T = 6 * torch.cuda.get_device_properties(0).multi_processor_count + 101
    window, ring, C, k = 128, 512, 700, 320
    win_row, comp_row = -(-(Dh + Dh // 32) // 16) * 16, -(-(Dh // 2 + Dh // 16) // 16) * 16
    u = torch.randn(Dh) / Dh ** 0.5
    win = torch.zeros(2, ring, win_row, dtype=torch.uint8)
    win[:, :, :Dh + Dh // 32] = codecs.kv_v41_encode(torch.randn(2, ring, Dh) * 1.5)
    comp = torch.zeros(2, C, comp_row, dtype=torch.uint8)
    comp[:, :, :Dh // 2 + Dh // 16] = codecs.kv_v41fp4_encode(torch.randn(2, C, Dh) + drift * torch.arange(C)[:, None] / C * u * 8)
    kvd, ckd = codecs.kv_v41_decode(win, Dh), codecs.kv_v41fp4_decode(comp, Dh)
    pos, region = (torch.arange(T) * 7 % 400).int(), (torch.arange(T) % 2).int()
    sel = torch.full((T, k), -1, dtype=torch.int32)
    cnt = torch.tensor([[0, 1, 37, 128, 129, 255, 320][r % 7] for r in range(T)], dtype=torch.int32)
    for r in range(T):
        sel[r, :cnt[r]] = torch.sort(torch.randperm(C)[:cnt[r]]).values.int()
    first = torch.where((cnt == 0) & (torch.arange(T) % 2 == 0), pos + 1, 0).int()         # (no window: no key at all)
    q = (torch.randn(T, Hl, Dh) * 0.5 + (drift > 0) * 40 * u * (torch.arange(Hl) % 2)[None, :, None]).bfloat16()
    sink = torch.randn(Hl) * 0.5
    freqs = torch.tensor([10000.0 ** (-2.0 * j / 64) for j in range(32)])
    dev = lambda t: t.to(DEV).contiguous()
    st = native.StatusWord(DEV)
    part = torch.zeros(1, device=DEV)                                  # (not read or written by this form)
    out = torch.zeros(T, Hl * Dh, device=DEV, dtype=torch.float16)
    native.call("tf_sparse_attention", dev(q), T, Hl, Dh, dev(pos), dev(region), dev(first), dev(win), ring * win_row, win_row,
                ring, window, dev(comp), C * comp_row, comp_row, dev(sel), k, dev(cnt), C, 1 / math.sqrt(Dh), 1, part, part,
                dev(sink), dev(freqs), 64, out, None, Hl * Dh, st.t)
    st.check()
    got = out.cpu().view(T, Hl, Dh).double()
    for r in range(T):
        p, rg = int(pos[r]), int(region[r])
        if first[r] > p:
            assert (got[r] == 0).all(), r
            continue
        nw = min(p + 1, window)
        keys = torch.cat([kvd[rg, [(p - nw + 1 + i) % ring for i in range(nw)]], ckd[rg, sel[r, :int(cnt[r])].long()]]).double()
        lg = torch.cat([q[r].double() @ keys.t() / math.sqrt(Dh), sink[:, None].double()], 1)
        o = apply_rope((torch.softmax(lg, -1)[:, :-1] @ keys)[None].float(), torch.tensor([p]), freqs, inverse=True)[0]
        assert _rel(got[r], o) < 1e-3, (r, _rel(got[r], o))


def test_sampling_kernels():
    torch.manual_seed(7)
    V, rows = 5000, 4
    lg = torch.randn(rows, V, device=DEV) * 3
    am = torch.zeros(rows, dtype=torch.int32, device=DEV)
    native.call("tf_argmax", lg, V, V, rows, am, None)
    assert am.cpu().tolist() == lg.argmax(-1).cpu().tolist()
    sb = native.lib().tf_rowstat_bytes()
    stat = torch.zeros(rows, sb, dtype=torch.uint8, device=DEV)
    st = native.StatusWord(DEV)
    T, top_p = 0.6, 0.95
    scr = torch.zeros(native.lib().tf_rowstats_scratch_bytes(rows), dtype=torch.uint8, device=DEV)
    native.call("tf_rowstats", lg, V, V, rows, T, top_p, stat, scr, st.t)
    assert int(scr.sum()) == 0          # every call leaves its scratch zeroed
    st.check()
    raw = stat.cpu().numpy().view(np.dtype([("m", "<f4"), ("thr", "<u4"), ("z", "<f8")]))
    pr = torch.softmax(lg.double().cpu() / T, -1)
    for r in range(rows):
        srt, _ = torch.sort(pr[r], descending=True)
        cs = torch.cumsum(srt, 0)
        n_in = int((cs < top_p).sum()) + 1
        mass = float(srt[:n_in].sum())
        z_total = float(torch.exp((lg[r].double().cpu() - lg[r].max().item()) / T).sum())
        assert abs(raw["z"][r][0] / z_total - mass) < 1e-6
    # plain sampling (g = 0): empirical law of the drawn tokens follows the nucleus distribution
    S = 4096
    lg1 = lg[:1].expand(S, V).contiguous()
    stat1 = stat[:1].expand(S, sb).contiguous()
    u = torch.rand(S, 2, dtype=torch.float64, device=DEV)
    R = torch.zeros(native.lib().tf_spec_verify_scratch_doubles(S, 0, V), dtype=torch.float64, device=DEV)
    w = torch.zeros(S, 1, dtype=torch.float64, device=DEV)
    nacc = torch.zeros(S, dtype=torch.int32, device=DEV)
    tok = torch.zeros(S, dtype=torch.int32, device=DEV)
    native.call("tf_spec_verify", lg1, None, stat1, None, None, u, S, 0, V, V, T, T, None, 0, R, w, nacc, tok, st.t)
    st.check()
    srt, idx = torch.sort(pr[0], descending=True)
    n_in = int((torch.cumsum(srt, 0) < top_p).sum()) + 1
    allowed = set(idx[:n_in].tolist())
    toks = tok.cpu().tolist()
    assert set(toks) <= allowed
    top = int(idx[0])
    want = float(srt[0] / srt[:n_in].sum())
    got = toks.count(top) / S
    assert abs(got - want) < 4 * math.sqrt(want * (1 - want) / S) + 1e-3


def test_block_verification_preserves_target_law():
    """Proposals from a draft law, verified against a target law: accepted/corrected first tokens
    must follow the target law (chi-square-style tolerance)."""
    torch.manual_seed(8)
    V, S, g = 64, 20000, 2
    tl = torch.randn(g + 1, V, device=DEV) * 1.5
    dl = tl[:g] + torch.randn(g, V, device=DEV) * 0.8
    T = 1.0
    sb = native.lib().tf_rowstat_bytes()
    st = native.StatusWord(DEV)
    tstat = torch.zeros(g + 1, sb, dtype=torch.uint8, device=DEV)
    dstat = torch.zeros(g, sb, dtype=torch.uint8, device=DEV)
    scr = torch.zeros(native.lib().tf_rowstats_scratch_bytes(g + 1), dtype=torch.uint8, device=DEV)
    native.call("tf_rowstats", tl, V, V, g + 1, T, 1.0, tstat, scr, st.t)
    native.call("tf_rowstats", dl, V, V, g, T, 1.0, dstat, scr, st.t)
    q = torch.softmax(dl.double(), -1)
    props = torch.stack([torch.multinomial(q[i], S, replacement=True) for i in range(g)], 1).int().contiguous()
    tlS = tl[None].expand(S, g + 1, V).contiguous()
    dlS = dl[None].expand(S, g, V).contiguous()
    u = torch.rand(S, g + 2, dtype=torch.float64, device=DEV)
    R = torch.zeros(native.lib().tf_spec_verify_scratch_doubles(S, g, V), dtype=torch.float64, device=DEV)
    w = torch.zeros(S, g + 1, dtype=torch.float64, device=DEV)
    nacc = torch.zeros(S, dtype=torch.int32, device=DEV)
    tok = torch.zeros(S, dtype=torch.int32, device=DEV)
    native.call("tf_spec_verify", tlS, dlS, tstat[None].expand(S, g + 1, sb).contiguous(),
                dstat[None].expand(S, g, sb).contiguous(), props, u, S, g, V, V, T, T, None, 0, R, w, nacc, tok, st.t)
    st.check()
    first = torch.where(nacc > 0, props[:, 0], tok).long().cpu()
    emp = torch.bincount(first, minlength=V).double() / S
    p0 = torch.softmax(tl[0].double().cpu(), -1)
    assert float((emp - p0).abs().max()) < 0.012
    assert 0.2 < float((nacc > 0).double().mean()) < 1.0


@pytest.mark.parametrize("Hl,drift", [(64, 0.0), (33, 0.0), (1, 0.0), (64, 12.0)])
def test_wide_sparse_attention_of_prefill_rows_on_tcgen05(Hl, drift):
    """Head dim 512, 64 rows or more of one split: 64-key chunks, the second contraction transposed.  Rows of one
    key, of exactly 64 and 65, of several chunks; ``drift`` makes later keys' scores grow, so that the reference
    maximum moves in some heads and their columns are rescaled.

    P and V are f16 (at most 2^-11 relative each, V exact), the output f16: within 1e-3 of the fp32 reference."""
    torch.manual_seed(18 + Hl)
    T, Dh, window, ring, C, k = 200, 512, 128, 512, 400, 320
    win_row, comp_row = Dh + Dh // 32, Dh // 2 + Dh // 16
    u = torch.randn(Dh) / Dh ** 0.5
    ramp = drift * torch.arange(C)[:, None] / C
    win = codecs.kv_v41_encode(torch.randn(2, ring, Dh) * 1.5)
    comp = codecs.kv_v41fp4_encode(torch.randn(2, C, Dh) + ramp * u * 8)
    kvd, ckd = codecs.kv_v41_decode(win, Dh), codecs.kv_v41fp4_decode(comp, Dh)
    pos = torch.cat([torch.arange(0, 100), torch.arange(300, 400)]).int()
    region = torch.cat([torch.zeros(100), torch.ones(100)]).int()
    sel = torch.full((T, k), -1, dtype=torch.int32)
    cnt = torch.zeros(T, dtype=torch.int32)
    for r in range(T):
        n = [0, 1, 37, 64, 129, 255, 320][r % 7]
        sel[r, :n] = torch.sort(torch.randperm(C)[:n]).values.int()
        cnt[r] = n
    q = (torch.randn(T, Hl, Dh) * 0.5 + (drift > 0) * 40 * u * (torch.arange(Hl) % 2)[None, :, None]).bfloat16()
    sink = torch.randn(Hl) * 0.5
    freqs = torch.tensor([10000.0 ** (-2.0 * j / 64) for j in range(32)])
    dev = lambda t: t.to(DEV).contiguous()
    st = native.StatusWord(DEV)
    from titanic_flash_41_b200.models.oracle import apply_rope
    for counts in (None, dev(cnt)):
        part_o, part_lse = torch.zeros(1, device=DEV), torch.zeros(1, device=DEV)      # (not read or written by this form)
        out = torch.zeros(T, Hl * Dh, device=DEV, dtype=torch.float16)
        outb = torch.zeros(T, Hl * Dh, device=DEV, dtype=torch.bfloat16)
        native.call("tf_sparse_attention", dev(q), T, Hl, Dh, dev(pos), dev(region), None, dev(win), ring * win_row,
                    win_row, ring, window, dev(comp), C * comp_row, comp_row, dev(sel), k, counts, C,
                    1 / math.sqrt(Dh), 1, part_o, part_lse, dev(sink), dev(freqs), 64, out, outb, Hl * Dh, st.t)
        st.check()
        got, gotb = out.cpu().view(T, Hl, Dh).double(), outb.cpu().view(T, Hl, Dh).double()
        for r in range(T):
            p, rg = int(pos[r]), int(region[r])
            nw = min(p + 1, window)
            Kmat = torch.cat([kvd[rg, [(p - nw + 1 + i) % ring for i in range(nw)]], ckd[rg, sel[r, :int(cnt[r])].long()]]).double()
            lg = torch.cat([q[r].double() @ Kmat.t() / math.sqrt(Dh), sink[:, None].double()], 1)
            o = apply_rope((torch.softmax(lg, -1)[:, :-1] @ Kmat)[None].float(), torch.tensor([p]), freqs, inverse=True)[0]
            assert _rel(got[r], o) < 1e-3 and _rel(gotb[r], o) < 4e-3, (r, _rel(got[r], o))


@pytest.mark.parametrize("world", [2, 4, 8])
def test_key_sharded_selection_equals_unsharded(world):
    """Scoring split over `world` key shards (run one after the other here) + gather + merge gives
    exactly the ids of the unsharded selection."""
    from titanic_flash_41_b200.parallel import key_sharded as KS
    torch.manual_seed(9)
    T, Hi, Di, C, k = 6, 8, 128, 5000, 256
    krow = Di // 2 + Di // 32
    keys = codecs.index_key_encode(torch.randn(1, C, Di)).to(DEV).contiguous()
    q = torch.randn(T, Hi, Di, device=DEV).bfloat16()
    w = torch.rand(T, Hi, device=DEV)
    region = torch.zeros(T, dtype=torch.int32, device=DEV)
    nvalid = torch.tensor([5000, 4097, 300, 0, 129, 2600], dtype=torch.int32, device=DEV)
    lds = 5120
    scores = torch.zeros(T, lds, device=DEV)
    native.call("tf_index_scores", q, w, region, nvalid, keys, C * krow, krow, T, Hi, Di, 2, scores, lds, 0, C)
    want = torch.full((T, k), -1, dtype=torch.int32, device=DEV)
    wcnt = torch.zeros(T, dtype=torch.int32, device=DEV)
    native.call("tf_topk_select", scores, lds, nvalid, k, want, wcnt, None, 0, T)
    parts = [KS.local_candidates(q, w, region, nvalid, keys, C * krow, krow, T, Hi, Di, 2,
                                 torch.zeros(T, lds, device=DEV), C, k, r, world) for r in range(world)]
    ids, cnt = KS.merge(torch.cat([p[0] for p in parts], 1), torch.cat([p[1] for p in parts], 1), k)
    torch.cuda.synchronize()
    assert torch.equal(cnt, wcnt)
    assert torch.equal(ids, want)


@pytest.mark.parametrize("T", [1, 5, 16, 19])
def test_router_logits_small_matches_fp32(T):
    torch.manual_seed(T)
    E_, d = 72, 1024
    x = torch.randn(T, d, device=DEV).bfloat16()
    gate = (torch.randn(E_, d, device=DEV) / 32).bfloat16()
    out = torch.zeros(T, E_, device=DEV)
    native.call("tf_router_logits_small", x, d, gate, out, E_, T, E_, d)
    again = torch.zeros(T, E_, device=DEV)
    native.call("tf_router_logits_small", x, d, gate, again, E_, T, E_, d)
    torch.cuda.synchronize()
    want = x.float() @ gate.float().t()
    assert (out - want).abs().max() <= 1e-4 * want.abs().max() + 1e-5
    assert torch.equal(out, again)


def test_route_group_many_experts_is_sorted_and_stable():
    torch.manual_seed(9)
    El, T, k, e_lo = 200, 16, 6, 56
    ids = torch.stack([torch.randperm(256, device=DEV)[:k] for _ in range(T)]).int().contiguous()
    n = T * k
    i32 = lambda m: torch.zeros(m, dtype=torch.int32, device=DEV)
    ge, gs, gc, ng, sp, nl = i32(El), i32(El), i32(El), i32(1), i32(n), i32(1)
    native.call("tf_route_group", ids, n, e_lo, e_lo + El, ge, gs, gc, ng, sp, nl)
    torch.cuda.synchronize()
    flat = ids.flatten().cpu() - e_lo
    local = [(int(e), i) for i, e in enumerate(flat.tolist()) if 0 <= e < El]
    want_sorted = [i for _, i in sorted(local)]                      # by expert, then pair order
    assert int(nl) == len(local) and sp[: len(local)].tolist() == want_sorted
    experts = sorted({e for e, _ in local})
    assert int(ng) == len(experts) and ge[: len(experts)].tolist() == experts
    counts = [sum(1 for e, _ in local if e == x) for x in experts]
    assert gc[: len(experts)].tolist() == counts
    starts = [sum(counts[:j]) for j in range(len(experts))]
    assert gs[: len(experts)].tolist() == starts


@pytest.mark.parametrize("d", [512, 4096])
def test_fused_boundary_equals_combine_then_norm_then_quantiser(d):
    """tf_add_norm_fused against tf_moe_combine + tf_add_norm + tf_quant_rows_mx8: the residual is
    bit-identical; the mean square is summed in another order, so a normalised value may land on the
    neighbouring bf16 value."""
    torch.manual_seed(12)
    T, k, El, e_lo = 9, 3, 6, 2
    x0 = torch.randn(T, d, device=DEV).bfloat16()
    y_pair = torch.randn(T * k, d, device=DEV)
    ids = torch.randint(0, 10, (T, k), device=DEV, dtype=torch.int32)
    wts = torch.rand(T, k, device=DEV)
    shared = torch.randn(T, d, device=DEV)
    w = (1 + 0.1 * torch.randn(d, device=DEV)).bfloat16()
    # separate kernels
    xa, delta = x0.clone(), torch.zeros(T, d, device=DEV)
    h16a, hba = torch.zeros(T, d, device=DEV, dtype=torch.float16), torch.zeros(T, d, device=DEV, dtype=torch.bfloat16)
    qa, sa = torch.zeros(T, d, dtype=torch.uint8, device=DEV), torch.zeros(T, d // 32, dtype=torch.uint8, device=DEV)
    native.call("tf_moe_combine", y_pair, ids, wts, shared, delta, T, d, k, e_lo, e_lo + El)
    native.call("tf_add_norm", xa, delta, 0, d, w, h16a, hba, None, None, T, d, 1e-6)
    native.call("tf_quant_rows_mx8", h16a, d, qa, sa, T, d)
    # one kernel
    xb = x0.clone()
    h16b, hbb, qb, sb = torch.zeros_like(h16a), torch.zeros_like(hba), torch.zeros_like(qa), torch.zeros_like(sa)
    native.call("tf_add_norm_fused", xb, None, y_pair, ids, wts, shared, k, e_lo, e_lo + El, w, h16b, hbb, qb, sb, T, d, 1e-6)
    torch.cuda.synchronize()
    assert torch.equal(xa, xb)
    for a, b_ in ((h16a, h16b), (hba, hbb)):
        assert (a.float() - b_.float()).abs().max() <= 0.01 * a.float().abs().max()
        assert (a == b_).float().mean() > 0.98
    deq = lambda q, s_: (q.view(torch.float8_e4m3fn).float().view(T, d // 32, 32) * torch.exp2(s_.float() - 127)[..., None])
    assert (deq(qa, sa) - deq(qb, sb)).abs().max() <= 0.07 * h16a.float().abs().max()
    assert (sa == sb).float().mean() > 0.98
    again = [torch.zeros_like(t) for t in (h16b, qb, sb)]
    xb2 = x0.clone()
    native.call("tf_add_norm_fused", xb2, None, y_pair, ids, wts, shared, k, e_lo, e_lo + El, w, again[0], None, again[1],
                again[2], T, d, 1e-6)
    torch.cuda.synchronize()
    assert torch.equal(again[0], h16b) and torch.equal(again[1], qb) and torch.equal(again[2], sb)   # run to run
    # plain delta source, no quantised copy
    xc, h16c = x0.clone(), torch.zeros_like(h16a)
    native.call("tf_add_norm_fused", xc, delta, None, None, None, None, 0, 0, 0, w, h16c, None, None, None, T, d, 1e-6)
    torch.cuda.synchronize()
    assert torch.equal(xc, xa) and (h16c == h16a).float().mean() > 0.98


@pytest.mark.parametrize("M", [3, 16, 27])
def test_router_topk_group_equals_the_two_launches(M):
    torch.manual_seed(M)
    E_, k, e_lo, El = 64, 6, 16, 32
    logits = torch.randn(M, E_, device=DEV)
    bias = torch.randn(E_, device=DEV) * 0.1
    i32 = lambda *s_: torch.zeros(*s_, dtype=torch.int32, device=DEV)
    out = []
    for fused in (False, True):
        ids, wts = i32(M, k), torch.zeros(M, k, device=DEV)
        ge, gs, gc, ng, sp, nl = i32(El), i32(El), i32(El), i32(1), i32(M * k), i32(1)
        if fused:
            native.call("tf_router_topk_group", logits, bias, None, None, -1, ids, wts, M, E_, k, 1, 1, 1.5, e_lo, e_lo + El,
                        ge, gs, gc, ng, sp, nl)
        else:
            native.call("tf_router_topk", logits, bias, None, None, -1, ids, wts, M, E_, k, 1, 1, 1.5)
            native.call("tf_route_group", ids, M * k, e_lo, e_lo + El, ge, gs, gc, ng, sp, nl)
        torch.cuda.synchronize()
        n, g = int(nl), int(ng)
        out.append((ids, wts, ge[:g].clone(), gs[:g].clone(), gc[:g].clone(), sp[:n].clone(), n, g))
    for a, b_ in zip(*out):
        assert torch.equal(a, b_) if isinstance(a, torch.Tensor) else a == b_


@pytest.mark.parametrize("T,n_max", [(4, 32768), (16, 20000), (3, 65536), (40, 30000), (36, 60000), (34, 70000)])
def test_topk_select_of_few_long_rows_matches_a_stable_sort(T, n_max):
    """A few long rows take the cluster-per-row kernel, more rows (or longer ones) the CTA-per-row
    kernel: same contract (exact, ties to the lower position, ids ascending, -1 padding, optional scores)."""
    torch.manual_seed(T)
    k, lds = 2048, n_max
    scores = (torch.randn(T, lds, device=DEV) * 0.3 + 5).relu()        # crowded exponents, like index scores
    scores[:, ::7] = scores[:, :1]                                      # many exact ties, some at the cut
    scores[0, :] = 1.25                                                 # a row of one value
    nvalid = torch.tensor([n_max, n_max - 13, 5000, 100][:T] + [n_max // 2 + i for i in range(max(0, T - 4))],
                          dtype=torch.int32, device=DEV)[:T]
    sel = torch.zeros(T, k, dtype=torch.int32, device=DEV)
    cnt = torch.zeros(T, dtype=torch.int32, device=DEV)
    osc = torch.zeros(T, k, device=DEV)
    native.call("tf_topk_select", scores, lds, nvalid, k, sel, cnt, osc, 100, T)
    torch.cuda.synchronize()
    for r in range(T):
        n = int(nvalid[r])
        s = scores[r, :n].cpu()
        got = sel[r].cpu().tolist()
        if n <= k:
            assert got == [100 + i for i in range(n)] + [-1] * (k - n) and int(cnt[r]) == n
            continue
        order = sorted(torch.sort(s, descending=True, stable=True).indices[:k].tolist())
        assert got == [100 + i for i in order] and int(cnt[r]) == k
        assert torch.equal(osc[r].cpu(), s[order])


@pytest.mark.parametrize("lds,k", [(33, 1), (1025, 1000), (4099, 512), (32800, 2048), (49152, 2048)])
def test_topk_select_of_many_rows_matches_a_stable_sort(lds, k):
    """One CTA per row, the row in shared memory: rows of one or two words of scores a thread, not a multiple of four,
    negative, infinite and equal scores (0 and -0 are different keys, so neither is drawn next to the other)."""
    T = 34
    gen = torch.Generator().manual_seed(lds)
    scores = torch.randn(T, lds, generator=gen)
    scores[:, 3::5] = scores[:, 2:3]
    scores[1] = -1.5
    scores[2, ::2] = -float("inf")
    scores[3, ::3] = float("inf")
    scores[4] = 2.0 + (torch.arange(lds) % 64) * 2.0 ** -21                  # equal but for the last bits
    nvalid = torch.tensor([lds - (i * 7) % (lds // 2 + 1) for i in range(T)], dtype=torch.int32)
    dev = scores.to(DEV)
    sel, cnt = torch.zeros(T, k, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)
    osc = torch.zeros(T, k, device=DEV)
    native.call("tf_topk_select", dev, lds, nvalid.to(DEV), k, sel, cnt, osc, 0, T)
    torch.cuda.synchronize()
    for r in range(T):
        n = int(nvalid[r])
        order = sorted(torch.sort(scores[r, :n], descending=True, stable=True).indices[:k].tolist())
        assert sel[r].cpu().tolist() == order + [-1] * (k - len(order)) and int(cnt[r]) == len(order)
        assert torch.equal(osc[r].cpu()[:len(order)], scores[r, order])


@pytest.mark.parametrize("T", [1, 4, 16, 27])
def test_router_topk_group_in_registers_equals_the_shared_memory_form(T):
    """256 experts or fewer: the single-launch kernel keeps each row in registers; selection bias per
    row (image-token rows use the second bias), same ids, weights and groups as the two launches."""
    torch.manual_seed(40 + T)
    E_, k, e_lo, El = 256, 6, 64, 64
    logits = torch.randn(T, E_, device=DEV)
    bias, bias_vl = torch.randn(E_, device=DEV) * 0.1, torch.randn(E_, device=DEV) * 0.1
    tokens = torch.randint(0, 3, (T,), dtype=torch.int32, device=DEV)
    i32 = lambda *s_: torch.zeros(*s_, dtype=torch.int32, device=DEV)
    out = []
    for fused in (False, True):
        ids, wts = i32(T, k), torch.zeros(T, k, device=DEV)
        ge, gs, gc, ng, sp, nl = i32(El), i32(El), i32(El), i32(1), i32(T * k), i32(1)
        if fused:
            native.call("tf_router_topk_group", logits, bias, bias_vl, tokens, 1, ids, wts, T, E_, k, 1, 1, 1.5, e_lo,
                        e_lo + El, ge, gs, gc, ng, sp, nl)
        else:
            native.call("tf_router_topk", logits, bias, bias_vl, tokens, 1, ids, wts, T, E_, k, 1, 1, 1.5)
            native.call("tf_route_group", ids, T * k, e_lo, e_lo + El, ge, gs, gc, ng, sp, nl)
        torch.cuda.synchronize()
        n, g = int(nl), int(ng)
        out.append((ids, wts, ge[:g].clone(), gs[:g].clone(), gc[:g].clone(), sp[:n].clone(), n, g))
    for a, b_ in zip(*out):
        assert torch.equal(a, b_) if isinstance(a, torch.Tensor) else a == b_


def test_mxfp4_to_fp8_block_conversion_is_exact_where_representable():
    """e2m1 x 2^e re-expressed as e4m3 with one power-of-two scale per 128 x 128 block: exact while a
    group's scale is within 2^-6 of the block's largest (e4m3 holds the shifted magnitudes), rounded
    to nearest below that, signs kept."""
    torch.manual_seed(21)
    E_, N, K = 2, 256, 512
    pk = torch.randint(0, 256, (E_, N, K // 2), device=DEV, dtype=torch.uint8)
    sc = torch.randint(118, 126, (E_, N, K // 32), device=DEV, dtype=torch.uint8)
    sc[0, :5, :3] = 100                                   # far below the block maximum: rounds towards zero
    out = torch.zeros(E_, N, K, dtype=torch.uint8, device=DEV)
    out_s = torch.zeros(E_ * N // 128, K // 128, device=DEV)
    native.call("tf_mxfp4_to_fp8_block", pk, sc, out, out_s, E_, N, K, 0, N)
    torch.cuda.synchronize()
    want = E.dequant_mxfp4(pk, sc)                        # [E, N, K] fp32
    got = out.view(torch.float8_e4m3fn).float().view(E_, N // 128, 128, K // 128, 128) \
        * out_s.view(E_, N // 128, 1, K // 128, 1)
    got = got.reshape(E_, N, K)
    close = sc.view(E_, N // 128, 128, K // 128, 4).float()
    top = close.amax(dim=(2, 4), keepdim=True)
    exact = ((top - close) <= 6).expand_as(close).reshape(E_, N, K // 32).repeat_interleave(32, dim=2)
    assert torch.equal(got[exact], want[exact])
    blk_max = want.abs().view(E_, N // 128, 128, K // 128, 128).amax(dim=(2, 4), keepdim=True).expand(
        E_, N // 128, 128, K // 128, 128).reshape(E_, N, K)
    assert ((got - want).abs() <= blk_max * 2.0 ** -9).all()
    nz = got != 0
    assert torch.equal(torch.signbit(got[nz]), torch.signbit(want[nz]))


def test_mx8_row_quantiser_matches_codec():
    """e4m3 values with one UE8M0 scale per 32 inputs: same bytes as the host codec."""
    torch.manual_seed(5)
    x = (torch.randn(7, 512, device=DEV) * torch.rand(7, 1, device=DEV) * 4).half()
    x[3, 64:96] = 0
    q = torch.zeros(7, 512, dtype=torch.uint8, device=DEV)
    s = torch.zeros(7, 16, dtype=torch.uint8, device=DEV)
    native.call("tf_quant_rows_mx8", x, 512, q, s, 7, 512)
    torch.cuda.synchronize()
    wq, ws = codecs.mxfp8_quant(x.float().cpu(), 32)
    assert torch.equal(s.cpu()[ws != 0], ws[ws != 0])          # an all-zero group may carry any scale
    back = q.view(torch.float8_e4m3fn).float().view(7, 16, 32) * torch.exp2(s.float() - 127)[..., None]
    assert (back.view(7, 512) - x.float()).abs().max() <= 0.07 * x.float().abs().max()
    assert torch.equal(q.cpu().view(7, 16, 32)[ws != 0], wq.view(torch.uint8).view(7, 16, 32)[ws != 0])


@pytest.mark.parametrize("dual,T", [(True, 16), (True, 5), (False, 16), (False, 3), (True, 24), (True, 32), (False, 24),
                                    (False, 32), (True, 17)])
def test_block_scaled_expert_gemv_matches_reference(dual, T):
    """MXFP4 weights x MXFP8 activations on tcgen05 block-scaled MMAs (scales applied by the tensor
    core) against fp32 math on the dequantised operands.  17..32 rows run the 32-column form."""
    from titanic_flash_41_b200.models import engine as E
    torch.manual_seed(7)
    El, N, K, k = 6, 256, 1024, 2
    w1 = torch.randn(El, N, K, device=DEV) * 0.1 * (1 + 3 * torch.rand(El, N, 1, device=DEV))
    w3 = torch.randn(El, N, K, device=DEV) * 0.1
    p1, s1 = E.quant_mxfp4_device(w1)
    p3, s3 = E.quant_mxfp4_device(w3)
    d1, d3 = E.dequant_mxfp4(p1, s1), E.dequant_mxfp4(p3, s3)
    ids = torch.stack([torch.randperm(El, device=DEV)[:k] for _ in range(T)]).int().contiguous()
    npairs = T * k
    i32 = lambda n: torch.zeros(n, dtype=torch.int32, device=DEV)
    ge, gs, gc, ng, sp, nl = i32(El), i32(El), i32(El), i32(1), i32(npairs), i32(1)
    native.call("tf_route_group", ids, npairs, 0, El, ge, gs, gc, ng, sp, nl)
    rows = T if dual else npairs                       # plain form: one activation row per sorted pair
    x = (torch.randn(rows, K, device=DEV) * (0.2 + 2 * torch.rand(rows, 1, device=DEV))).half()
    xq = torch.zeros(rows, K, dtype=torch.uint8, device=DEV)
    xs = torch.zeros(rows, K // 32, dtype=torch.uint8, device=DEV)
    native.call("tf_quant_rows_mx8", x, K, xq, xs, rows, K)
    xd = (xq.view(torch.float8_e4m3fn).float().view(rows, K // 32, 32)
          * torch.exp2(xs.float() - 127)[..., None]).view(rows, K)
    st = native.StatusWord(DEV)
    if dual:
        y = torch.zeros(npairs, N, device=DEV, dtype=torch.float16)
    else:
        y = torch.zeros(npairs, N, device=DEV)
    y8 = torch.zeros(npairs, N, dtype=torch.uint8, device=DEV)
    y8s = torch.zeros(npairs, N // 32, dtype=torch.uint8, device=DEV)
    native.call("tf_moe_gemv_mx", p1, p3 if dual else None, s1, s3 if dual else None, El, xq, xs, rows, y, N,
                y8 if dual else None, y8s if dual else None, N, K, k, ge, gs, gc, ng, sp, min(El, npairs),
                10.0 if dual else 0.0, 0, 0, T, st.t)
    torch.cuda.synchronize()
    st.check()
    if dual:
        # the MXFP8 copy of the fused output equals quantising the f16 rows (up to f16 rounding of the input)
        back = (y8.view(torch.float8_e4m3fn).float().view(npairs, N // 32, 32)
                * torch.exp2(y8s.float() - 127)[..., None]).view(npairs, N)
        assert (back - y.float()).abs().max() <= 0.07 * y.float().abs().max() + 1e-3
    order = sp.tolist()
    for pos, pair in enumerate(order):
        t, j = divmod(pair, k)
        e = int(ids[t, j])
        if dual:
            a = d1[e] @ xd[t]
            up = (d3[e] @ xd[t]).clamp(-10, 10)
            want = torch.nn.functional.silu(a.clamp(max=10)) * up
            got = y[pos].float()                       # fused form writes rows in sorted pair order
            tol = 2e-3 * want.abs().max() + 2e-3
        else:
            want = d1[e] @ xd[pos]
            got = y[pair]
            tol = 1e-3 * want.abs().max() + 1e-4
        assert (got - want).abs().max() <= tol, (pos, pair, float((got - want).abs().max()), float(want.abs().max()))


def test_two_level_candidates_match_dense_selection():
    """Sparse scores equal the dense ones at the candidate keys, and selecting among the published
    blocks gives the dense top-k whenever all of it lies inside them."""
    from titanic_flash_41_b200.ops import two_level as TL
    torch.manual_seed(11)
    T, Hi, Di, C, k = 5, 8, 128, 4000, 64
    krow = Di // 2 + Di // 32
    keys = codecs.index_key_encode(torch.randn(1, C, Di)).to(DEV).contiguous()
    q = torch.randn(T, Hi, Di, device=DEV).bfloat16()
    w = torch.rand(T, Hi, device=DEV)
    region = torch.zeros(T, dtype=torch.int32, device=DEV)
    nvalid = torch.tensor([4000, 3001, 517, 64, 9], dtype=torch.int32, device=DEV)
    lds = 4096
    scores = torch.zeros(T, lds, device=DEV)
    native.call("tf_index_scores", q, w, region, nvalid, keys, C * krow, krow, T, Hi, Di, 1, scores, lds, 0, C)
    want = torch.full((T, k), -1, dtype=torch.int32, device=DEV)
    wcnt = torch.zeros(T, dtype=torch.int32, device=DEV)
    native.call("tf_topk_select", scores, lds, nvalid, k, want, wcnt, None, 0, T)
    cand = TL.publish(scores[:, :C], nvalid, n_blocks=128, T=T)
    assert cand.shape == (T, 1024)
    for r in range(T):
        c = cand[r][cand[r] >= 0]
        assert bool((c[1:] > c[:-1]).all()) and int(c.max()) < int(nvalid[r])
    sc = torch.empty(T, cand.shape[1], device=DEV)
    native.call("tf_index_scores_sparse", q, w, region, cand, cand.stride(0), keys, C * krow, krow, T, Hi, Di,
                cand.shape[1], sc, cand.shape[1])
    torch.cuda.synchronize()
    ok = cand >= 0
    dense_at = torch.gather(scores, 1, cand.clamp_min(0).long())
    assert (sc[ok] - dense_at[ok]).abs().max() <= 1e-3 * dense_at[ok].abs().max() + 1e-5
    assert bool(torch.isinf(sc[~ok]).all())
    ids, cnt = TL.consume(q, w, region, cand, keys, C * krow, krow, T, Hi, Di, k)
    assert torch.equal(cnt, wcnt)
    # the best 64 keys sit in the best 128 blocks of 8 (every top key's block maximum is at least its own
    # score); the two scorings may only disagree about keys that tie with the cut within rounding
    for r in range(T):
        a, b = set(ids[r][ids[r] >= 0].tolist()), set(want[r][want[r] >= 0].tolist())
        if a != b:
            cut = min(float(scores[r, i]) for i in b)
            assert all(abs(float(scores[r, i]) - cut) <= 1e-3 * abs(cut) + 1e-5 for i in a ^ b), r


@pytest.mark.parametrize("T,d,kind", [(1, 128, None), (3, 4096, "f32"), (5, 5120, "bf16"), (2, 8192, "f32"), (2, 8320, "f32"), (70, 384, "bf16")])
def test_add_norm_vector_form(T, d, kind):
    """One and two 16-byte pieces a thread (the second ragged at 5120), a width beyond the vector form, and both kinds of delta.

    The residual is one bf16 rounding of an fp32 sum (exact match); the normalised row one bf16 rounding (2^-8) of
    values whose fp32 mean square has an error far below that."""
    torch.manual_seed(d + T)
    x = torch.randn(T, d, device=DEV).bfloat16()
    delta = None if kind is None else torch.randn(T, d, device=DEV).to(torch.float32 if kind == "f32" else torch.bfloat16)
    w = (1 + 0.1 * torch.randn(d, device=DEV)).bfloat16()
    h16, hb = torch.zeros(T, d, device=DEV, dtype=torch.float16), torch.zeros(T, d, device=DEV, dtype=torch.bfloat16)
    res = x.clone() if delta is None else (x.float() + delta.float()).bfloat16()
    native.call("tf_add_norm", x, delta, 1 if kind == "bf16" else 0, d, w, h16, hb, None, None, T, d, 1e-6)
    assert torch.equal(x, res)
    want = res.double() * torch.rsqrt(res.double().pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert ((hb.double() - want).abs() <= 2.0 ** -8 * 1.01 * want.abs() + 1e-30).all() and torch.equal(h16, hb.half())


@pytest.mark.parametrize("T", [1, 4, 5, 8, 9, 17, 32])
@pytest.mark.parametrize("E_,d", [(256, 4096), (33, 8), (384, 5120)])
def test_router_logits_row_forms(T, E_, d):
    """The three row forms and several passes, an odd number of experts, fewer 16-byte steps than warps: fp32 sums
    of exact products, against fp64."""
    torch.manual_seed(T + E_)
    x, gate = torch.randn(T, d, device=DEV).bfloat16(), torch.randn(E_, d, device=DEV).bfloat16()
    out = torch.full((T, E_ + 1), 3.0, device=DEV)
    native.call("tf_router_logits_small", x, d, gate, out, E_ + 1, T, E_, d)
    want = x.double() @ gate.double().t()
    assert float((out[:, :E_].double() - want).abs().max()) < 1e-5 * d ** 0.5 + 1e-6 and (out[:, E_] == 3.0).all()


@pytest.mark.parametrize("T,Hi,C,lo,hi", [(33, 8, 300, 0, 300), (70, 8, 2600, 0, 2600), (64, 16, 1000, 128, 900), (45, 32, 700, 0, 700),
                                          (40, 64, 129, 0, 129), (320, 8, 9000, 0, 9000)])
def test_index_scores_of_prefill_rows_on_tcgen05(T, Hi, C, lo, hi):
    """Row tiles of 32, 16, 8 and 4 rows with a ragged last one, key tiles that end inside, at and one past 128 keys, a
    shard of the keys, causal counts (rows without a valid key included): scores against fp64, -inf from a row's
    count to the end of the shard, nothing written outside it.

    Operands are exact in f16; a score is a sum over heads of fp32 sums of 128 products: 1e-5 of its magnitude."""
    torch.manual_seed(T + Hi)
    Di, lds = 128, C + 40
    enc = codecs.index_key_encode(torch.randn(1, C, Di))
    kd = codecs.index_key_decode(enc, Di)[0].to(DEV).double()
    keys = enc.to(DEV).contiguous()
    krow = enc.shape[-1]
    q, w = torch.randn(T, Hi, Di, device=DEV).bfloat16(), torch.randn(T, Hi, device=DEV)
    region = torch.zeros(T, dtype=torch.int32, device=DEV)
    nvalid = torch.linspace(0, C, T, device=DEV).int()
    scores = torch.full((T, lds), 7.0, device=DEV)
    st = native.StatusWord(DEV)
    native.call("tf_index_scores_rows", q, w, region, nvalid, keys, C * krow, krow, T, Hi, Di, 32, scores, lds, lo, hi, st.t)
    st.check()
    s = torch.einsum("thd,cd->thc", q.double(), kd).relu()
    want, mag = (s * w.double()[:, :, None]).sum(1), (s * w.double().abs()[:, :, None]).sum(1)
    col = torch.arange(C, device=DEV)[None, :]
    live = (col < nvalid[:, None]) & (col >= lo) & (col < hi)
    err = (scores[:, :C].double() - want).abs()
    assert bool((err[live] <= 1e-5 * mag[live] + 1e-5).all()), float((err / (mag + 1))[live].max())
    dead = (col >= nvalid[:, None]) & (col >= lo) & (col < hi)
    assert bool((scores[:, :C][dead] == -float("inf")).all())
    assert bool((scores[:, hi:] == 7.0).all()) and bool((scores[:, :lo] == 7.0).all())


@pytest.mark.parametrize("scales", [(120, 127), (103, 104), (142, 143), (0, 110)])
def test_index_scores_of_prefill_rows_take_every_block_scale(scales):
    """Key blocks whose scales lie on both sides of the line between the f16 product and the fp32 one (2^-23 to 2^15): a key
    element is its value rounded once to f16, whichever way it is formed.  Values of one half where larger ones would
    overflow f16; queries exact in f16; the bound is that of the test above."""
    torch.manual_seed(sum(scales))
    T, Hi, Di, C = 40, 8, 128, 300
    nib = torch.randint(0, 16, (C, Di)) if max(scales) < 140 else torch.randint(0, 2, (C, Di)) + 8 * torch.randint(0, 2, (C, Di))
    sc = torch.tensor(scales)[torch.randint(0, 2, (C, Di // 32))]
    keys = torch.cat([nib[:, 0::2] | nib[:, 1::2] << 4, sc], 1).to(torch.uint8).to(DEV).contiguous()
    val = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, 0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64)[nib]
    kd = (val * torch.exp2(sc.double() - 127).repeat_interleave(32, 1)).half().double().to(DEV)
    q = (torch.randint(-64, 65, (T, Hi, Di), device=DEV) / 16.0).bfloat16()
    w = torch.randn(T, Hi, device=DEV)
    region, nvalid = torch.zeros(T, dtype=torch.int32, device=DEV), torch.full((T,), C, dtype=torch.int32, device=DEV)
    scores, st = torch.zeros(T, C, device=DEV), native.StatusWord(DEV)
    native.call("tf_index_scores_rows", q, w, region, nvalid, keys, C * 68, 68, T, Hi, Di, 32, scores, C, 0, C, st.t)
    st.check()
    s = torch.einsum("thd,cd->thc", q.double(), kd)
    size = torch.einsum("thd,cd->thc", q.double().abs(), kd.abs())
    want, mag = (s.relu() * w.double()[:, :, None]).sum(1), (size * w.double().abs()[:, :, None]).sum(1)
    assert bool(((scores.double() - want).abs() <= 1e-5 * mag).all())


def test_index_scores_and_router_logits_round_no_more_than_the_kernels_they_replaced():
    """Error against fp64 (2-norm over 2-norm): 6.4e-8 for the index scores of 64 heads and 8.06e-8 for the router logits of
    256 x 4,096 with the kernels before; one chain over all heads or warps gives 1.05e-7 and 8.4e-8.  The bounds lie between."""
    torch.manual_seed(5)
    T, Hi, Di, C = 200, 64, 128, 4000
    enc = codecs.index_key_encode(torch.randn(1, C, Di))
    keys, kd = enc.to(DEV).contiguous(), codecs.index_key_decode(enc, Di)[0].to(DEV).double()
    q, w = torch.randn(T, Hi, Di, device=DEV).bfloat16(), torch.randn(T, Hi, device=DEV)
    region, nvalid = torch.zeros(T, dtype=torch.int32, device=DEV), torch.full((T,), C, dtype=torch.int32, device=DEV)
    scores, st = torch.zeros(T, C, device=DEV), native.StatusWord(DEV)
    native.call("tf_index_scores_rows", q, w, region, nvalid, keys, C * enc.shape[-1], enc.shape[-1], T, Hi, Di, 32, scores, C, 0, C, st.t)
    st.check()
    want = (torch.einsum("thd,cd->thc", q.double(), kd).relu() * w.double()[:, :, None]).sum(1)
    assert float((scores.double() - want).norm() / want.norm()) < 8e-8
    err = mag = 0.0
    for _ in range(20):
        x, gate = torch.randn(32, 4096, device=DEV).bfloat16(), torch.randn(256, 4096, device=DEV).bfloat16()
        out = torch.zeros(32, 256, device=DEV)
        native.call("tf_router_logits_small", x, 4096, gate, out, 256, 32, 256, 4096)
        want = x.double() @ gate.double().t()
        err, mag = err + float((out.double() - want).pow(2).sum()), mag + float(want.pow(2).sum())
    assert (err / mag) ** 0.5 < 8.1e-8


@pytest.mark.parametrize("T,n,lds,k", [(33, 5000, 5000, 512), (33, 4097, 4099, 2048), (40, 49152, 49152, 2048), (34, 50000, 50000, 33), (2, 3000, 4096, 1)])
def test_topk_select_rows_edges(T, n, lds, k):
    """Rows in shared memory up to its limit, one past it, strides off the vector grain, k of one, all three digits
    deciding: negative, equal and nearly equal scores."""
    torch.manual_seed(n)
    scores = torch.randn(T, lds, device=DEV)
    scores[0] = -scores[0].abs() - 1
    scores[1] = 1.0 + torch.randint(0, 3, (lds,), device=DEV) * 2.0 ** -23
    nvalid = torch.full((T,), n, dtype=torch.int32, device=DEV)
    sel, cnt = torch.zeros(T, k, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)
    native.call("tf_topk_select", scores, lds, nvalid, k, sel, cnt, None, 0, T)
    for r in range(T):
        order = torch.sort(scores[r, :n].cpu(), descending=True, stable=True).indices[:k].sort().values
        assert torch.equal(sel[r].cpu().long(), order) and int(cnt[r]) == k


@pytest.mark.parametrize("T,R,ld,kind", [(1, 1280, 1408, "f32"), (33, 40, 41, "f32"), (5, 1000, 1536, "bf16")])
def test_rms_of_projection_columns(T, R, ld, kind):
    """A column range of wider rows, widths off the block size: f16 rounding (2^-11) of an fp32 normalisation."""
    torch.manual_seed(R)
    x = torch.randn(T, ld, device=DEV).to(torch.float32 if kind == "f32" else torch.bfloat16)
    w = (1 + 0.1 * torch.randn(R, device=DEV)).bfloat16()
    out = torch.zeros(T, R, device=DEV, dtype=torch.float16)
    native.call("tf_rms_cols", x[:, ld - R:], 0 if kind == "f32" else 2, ld, w, out, T, R, 1e-6)
    v = x[:, ld - R:].double()
    want = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert ((out.double() - want).abs() <= 2.0 ** -11 * 1.01 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("M,G,R,K", [(1, 8, 128, 384), (24, 3, 1024, 512), (32, 2, 256, 128)])
def test_block_diagonal_gemv(M, G, R, K):
    """Every block reads its own K activations and writes its own columns (one tile, several tiles per block); f16 out."""
    torch.manual_seed(M)
    ws = [E.quant_fp8_device(torch.randn(R, K, device=DEV) * 0.1 * (g + 1)) for g in range(G)]
    L = E.LayerWeights(wo_a=ws)
    E.stack_blocks(L)
    assert all(torch.equal(a.q.view(torch.uint8), b_.q.view(torch.uint8)) and torch.equal(a.s, b_.s) for a, b_ in zip(ws, L.wo_a))
    x = torch.randn(M, G * K + 8, device=DEV).half()
    out = torch.zeros(M, G * R, device=DEV, dtype=torch.float16)
    native.call("tf_smallm_gemm_blocks", L.wo_a_all.q, L.wo_a_all.s, x, x.stride(0), out, out.stride(0), G, R, K, M)
    for g in range(G):
        want = x[:, g * K:(g + 1) * K].double() @ E.dequant_fp8(ws[g]).double().t()
        assert float((out[:, g * R:(g + 1) * R].double() - want).norm() / want.norm()) < 2.0 ** -11 + 1e-5


@pytest.mark.parametrize("T,d,k,shared", [(1, 128, 1, False), (3, 4096, 6, True), (5, 1280, 9, True), (2, 5120, 8, False)])
def test_fused_boundary_row_form(T, d, k, shared):
    """One piece a thread (narrow and full rows), more experts than are requested at once, and a width beyond it: residual
    exact against fp32 sums in slot order, the normalised row one bf16 rounding (2^-8), its MXFP8 form exact."""
    torch.manual_seed(d + k)
    El = 5
    x = torch.randn(T, d, device=DEV).bfloat16()
    y, wts = torch.randn(T * k, d, device=DEV), torch.rand(T, k, device=DEV)
    ids = torch.randint(0, 8, (T, k), dtype=torch.int32, device=DEV)
    sh = torch.randn(T, d, device=DEV) if shared else None
    w = (1 + 0.1 * torch.randn(d, device=DEV)).bfloat16()
    h16, hb = torch.zeros(T, d, dtype=torch.float16, device=DEV), torch.zeros(T, d, dtype=torch.bfloat16, device=DEV)
    x8, x8s = torch.zeros(T, d, dtype=torch.uint8, device=DEV), torch.zeros(T, d // 32, dtype=torch.uint8, device=DEV)
    own = ((ids >= 2) & (ids < 2 + El)).float()[:, :, None]
    sums = (y.view(T, k, d).double() * (wts[:, :, None] * own).double()).sum(1) + (sh.double() if shared else 0.0)
    want_x = x.double() + sums
    native.call("tf_add_norm_fused", x, None, y, ids, wts, sh, k, 2, 2 + El, w, h16, hb, x8, x8s, T, d, 1e-6)
    assert ((x.double() - want_x).abs() <= 2.0 ** -8 * 1.01 * want_x.abs() + 1e-5).all()
    want = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert ((hb.double() - want).abs() <= 2.0 ** -8 * 1.01 * want.abs() + 1e-30).all() and torch.equal(h16, hb.half())
    q, s = torch.zeros_like(x8), torch.zeros_like(x8s)
    native.call("tf_quant_rows_mx8", h16, d, q, s, T, d)
    assert torch.equal(q, x8) and torch.equal(s, x8s)


@pytest.mark.parametrize("T,d,m", [(1, 8, 1), (33, 2056, 3), (70, 5120, 4)])
def test_expanded_rows_are_copies(T, d, m):
    """Fewer and more pieces than threads, a ragged last round; rows behind the last one stay."""
    src = torch.randn(T, d, device=DEV).bfloat16()
    out = torch.full((T + 1, m, d), 3.0, device=DEV, dtype=torch.bfloat16)
    native.call("tf_expand_rows", src, out, T, d, m)
    assert torch.equal(out[:T], src[:, None, :].expand(T, m, d)) and bool((out[T] == 3.0).all())
