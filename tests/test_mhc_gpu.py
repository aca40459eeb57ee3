"""mHC boundary kernels against the oracle's fp32 functions."""
import pytest
import torch

from titanic_flash_41_b200.models import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,d", [(1, 4, 512), (13, 4, 1280), (5, 2, 256)])
def test_prepare_and_post_match_oracle(T, H, d):
    from titanic_flash_41_b200.ops.mhc import HcBoundary
    dev = "cuda"
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, H, d, generator=g).bfloat16()
    fn = torch.randn(H * (2 + H), H * d, generator=g) * 0.05
    base = torch.randn(H * (2 + H), generator=g) * 0.3
    scale = torch.tensor([0.7, 1.3, 0.9])
    nw = (1 + 0.1 * torch.randn(d, generator=g)).bfloat16()
    hb = HcBoundary(fn.to(dev), base.to(dev), scale.to(dev), H, d, iters=20, eps=1e-6, rms_eps=1e-6)
    v, h16 = hb.prepare(x.to(dev), nw.to(dev))
    pre, post, comb = oracle.hc_coefficients(x.float(), fn, base, scale, 20, 1e-6, 1e-6)
    gp, gq, gc = (t.float().cpu() for t in hb.coefficients(T))
    assert (gp - pre).abs().max() < 2e-3 and (gq - post).abs().max() < 2e-3 and (gc - comb).abs().max() < 2e-3
    want_v = oracle.hc_collapse(x.float(), pre)
    assert (v.float().cpu() - want_v).abs().max() < 0.03 * want_v.abs().max() + 1e-2
    want_h = oracle.rmsnorm(want_v.bfloat16().float(), nw.float(), 1e-6)
    assert (h16.float().cpu() - want_h).abs().max() < 0.05
    a = torch.randn(T, d, generator=g)
    y = hb.finish(x.to(dev), a.to(dev)).float().cpu()
    want_y = oracle.hc_post(x.float(), a, post, comb)
    assert (y - want_y).abs().max() < 0.03 * want_y.abs().max() + 1e-2


@pytest.mark.parametrize("T,H,d", [(1, 4, 5120), (37, 3, 136), (38, 4, 5120), (100, 4, 1000), (65, 2, 72), (50, 1, 64), (40, 4, 100), (40, 4, 10304)])
def test_prepare_post_and_head_over_both_forms(T, H, d):
    """One row and sixteen rows per cluster (the line is at 37 rows), ragged last clusters, widths that do not
    divide into eight slices, rows too wide for sixteen at once, and a width off the vector grain (general kernel; no head form).

    fp32 sums of n = H d products in two orders differ by at most about 2 n 2^-24 of the sum of magnitudes, and
    in practice by its square root: far below 1e-4 of a mix here; stored rows carry bf16 rounding, 2^-8 relative at most."""
    from titanic_flash_41_b200.ops import native
    from titanic_flash_41_b200.ops.mhc import HcBoundary
    dev = "cuda"
    g = torch.Generator().manual_seed(T * d)
    x = torch.randn(T, H, d, generator=g).bfloat16()
    fn = torch.randn(H * (2 + H), H * d, generator=g) * 0.05
    base = torch.randn(H * (2 + H), generator=g) * 0.3
    scale = torch.tensor([0.7, 1.3, 0.9])
    nw = (1 + 0.1 * torch.randn(d, generator=g)).bfloat16()
    hb = HcBoundary(fn.to(dev), base.to(dev), scale.to(dev), H, d, iters=20, eps=1e-6, rms_eps=1e-6)
    v, h16 = hb.prepare(x.to(dev), nw.to(dev))
    pre, post, comb = (t.double() for t in oracle.hc_coefficients(x.float(), fn, base, scale, 20, 1e-6, 1e-6))
    for got, want in zip(hb.coefficients(T), (pre, post, comb)):
        assert (got.double().cpu() - want).abs().max() < 2e-4

    def bf16_close(got, want):                  # one bf16 rounding, plus the coefficients' 2e-4
        return ((got.double().cpu() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-3).all()
    want_v = (x.double() * pre[:, :, None]).sum(1)
    assert bf16_close(v, want_v)
    vb = v.double().cpu()
    want_h = vb * torch.rsqrt(vb.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double()
    assert ((h16.double().cpu() - want_h).abs() <= 2.0 ** -10 * want_h.abs() + 1e-4).all()
    a = torch.randn(T, d, generator=g)
    y = hb.finish(x.to(dev), a.to(dev))
    want_y = post[:, :, None] * a.double()[:, None] + torch.einsum("thc,thd->tcd", comb, x.double())
    assert bf16_close(y, want_y)
    if d % 8:
        return
    hfn, hbase, hscale = fn[:H].contiguous().to(dev), base[:H].contiguous().to(dev), scale[:1].to(dev)
    hv, hm = (torch.empty(T, d, dtype=torch.bfloat16, device=dev) for _ in range(2))
    hh, hbf = torch.empty(T, d, dtype=torch.float16, device=dev), torch.empty(T, d, dtype=torch.bfloat16, device=dev)
    native.call("tf_hc_head", x.to(dev), hfn, hbase, hscale, hv, hm, nw.to(dev), hh, hbf, T, H, d, 1e-6, 1e-6)
    flat = x.double().reshape(T, -1)
    mixes = (flat @ fn[:H].double().t()) * torch.rsqrt(flat.pow(2).mean(-1, keepdim=True) + 1e-6)
    hp = torch.sigmoid(mixes * 0.7 + base[:H].double()) + 1e-6
    assert bf16_close(hv, (x.double() * hp[:, :, None]).sum(1)) and bf16_close(hm, x.double().mean(1))
    hvb = hv.double().cpu()
    want = hvb * torch.rsqrt(hvb.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double()
    assert bf16_close(hbf, want) and torch.equal(hh, hbf.half())


def test_boundaries_of_two_widths_from_several_threads():
    """Host threads with streams of their own, sixteen-row clusters of 82 KB in one half and of 164 KB in the other, launched
    back to back: a limit set to the bytes of each launch would be lowered by one thread between another's set and launch."""
    import threading
    from titanic_flash_41_b200.ops import native
    from titanic_flash_41_b200.ops.mhc import HcBoundary
    H, rows, errors = 4, 40, []
    lib = native.lib()
    start = threading.Barrier(8)

    def work(d, seed):
        try:
            g = torch.Generator(device="cuda").manual_seed(seed)
            x = torch.randn(rows, H, d, generator=g, device="cuda").bfloat16()
            fn = torch.randn(H * (2 + H), H * d, generator=g, device="cuda") * 0.05
            hb = HcBoundary(fn, torch.zeros(H * (2 + H), device="cuda"), torch.ones(3, device="cuda"), H, d)
            first, v = hb.prepare(x)[0], torch.empty(rows, d, dtype=torch.bfloat16, device="cuda")
            stream = torch.cuda.Stream()
            torch.cuda.synchronize()
            start.wait()
            args = [x.data_ptr(), hb.fn.data_ptr(), hb.base.data_ptr(), hb.scale.data_ptr(), hb._coef.data_ptr(), v.data_ptr(),
                    None, None, None, rows, H, d, 1, 1e-6, 1e-6, stream.cuda_stream]
            refused = sum(lib.tf_hc_prepare(*args) != 0 for _ in range(4000))
            torch.cuda.synchronize()
            errors.append((refused, bool(torch.equal(v, first))))
        except Exception as e:
            errors.append(repr(e))
    torch.zeros(1, device="cuda")
    threads = [threading.Thread(target=work, args=((5120, 10240)[i % 2], i)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == [(0, True)] * 8


@pytest.mark.parametrize("T,H,d,off", [(3, 4, 100, 0), (1, 3, 41, 0), (40, 2, 1028, 0), (5, 4, 512, 1), (2, 4, 128, 3)])
def test_head_collapse_of_any_width_and_alignment(T, H, d, off):
    """Widths that eight does not divide and weights that start ``off`` floats behind a 16-byte boundary (the general
    kernel), against fp64; mixes and bounds as in the test of the cluster forms."""
    from titanic_flash_41_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(T * d)
    x = torch.randn(T, H, d, generator=g, device="cuda").bfloat16()
    fn = torch.zeros(H * H * d + off, device="cuda")[off:].view(H, H * d).copy_(torch.randn(H, H * d, generator=g, device="cuda") * 0.05)
    base, scale = torch.randn(H, generator=g, device="cuda") * 0.3, torch.full((1,), 0.7, device="cuda")
    nw = (1 + 0.1 * torch.randn(d, generator=g, device="cuda")).bfloat16()
    v, mean, hb = (torch.zeros(T, d, dtype=torch.bfloat16, device="cuda") for _ in range(3))
    h16 = torch.zeros(T, d, dtype=torch.float16, device="cuda")
    native.call("tf_hc_head", x, fn, base, scale, v, mean, nw, h16, hb, T, H, d, 1e-6, 1e-6)
    flat = x.double().reshape(T, -1)
    pre = torch.sigmoid(flat @ fn.double().t() * torch.rsqrt(flat.pow(2).mean(-1, keepdim=True) + 1e-6) * 0.7 + base.double()) + 1e-6

    def bf16_close(got, want):                  # one bf16 rounding, plus the coefficients' 2e-4
        return bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-3).all())
    assert bf16_close(v, (x.double() * pre[:, :, None]).sum(1)) and bf16_close(mean, x.double().mean(1))
    vd = v.double()
    want = vd * torch.rsqrt(vd.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double()
    assert bf16_close(hb, want) and torch.equal(h16, hb.half())
    v2 = torch.zeros_like(v)
    native.call("tf_hc_head", x, fn, base, scale, v2, None, None, None, None, T, H, d, 1e-6, 1e-6)      # without mean and norm
    assert torch.equal(v, v2)


@pytest.mark.parametrize("T", [24, 200])
def test_mixes_of_wide_rows_round_no_more_than_fp32_sums(T):
    """20,480 columns, 2-norm error of the collapse weights against fp64: fp32 multiply-adds (one row a cluster) 1.3e-7, sixteen rows
    on the tensor cores with each step's sum added in fp32 1.1e-7.  All steps in the tensor cores' own accumulator, which
    truncates what it adds, gave 5.4e-7: the bound lies between."""
    from titanic_flash_41_b200.ops.mhc import HcBoundary
    H, d = 4, 5120
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, H, d, generator=g).bfloat16()
    fn = torch.randn(H * (2 + H), H * d, generator=g) * 0.05
    base, scale = torch.randn(H * (2 + H), generator=g) * 0.3, torch.tensor([0.7, 1.3, 0.9])
    hb = HcBoundary(fn.cuda(), base.cuda(), scale.cuda(), H, d)
    hb.prepare(x.cuda())
    flat = x.double().reshape(T, -1)
    mixes = (flat @ fn[:H].double().t()) * torch.rsqrt(flat.pow(2).mean(-1, keepdim=True) + 1e-6)
    pre = torch.sigmoid(mixes * scale[0].double() + base[:H].double()) + 1e-6
    got = hb.coefficients(T)[0].double().cpu()
    assert float((got - pre).norm() / pre.norm()) < 2.5e-7
