"""Image input planning / patchify (CPU) and the device vision tower against its fp32 oracle (GPU)."""
import io
import math

import numpy as np
import pytest
import torch

from titanic_flash_41_b200.api import vision_input as VI
from titanic_flash_41_b200.config import VisionConfig


def test_plan_token_budget_and_padding():
    p = VI.Plan.new(640, 480)
    assert p.width % 14 == 0 and p.height % 14 == 0 and p.tokens == p.llm_height * (p.llm_width + 1) + 2
    assert p.tokens <= 1024 and p.resize_width <= p.width and p.resize_height <= p.height
    big = VI.Plan.new(8000, 6000)
    assert big.tokens <= 1024 and big.vit_height * big.vit_width <= 9198
    tall = VI.Plan.new(50, 20000)
    assert tall.tokens <= 1024
    small = VI.Plan.new(32, 32)                  # tiny images are scaled up to the minimum area first
    assert small.width * small.height >= 500 * 500
    with pytest.raises(ValueError):
        VI.Plan.new(0, 10)


def test_prepare_patch_layout_and_cache():
    from PIL import Image
    rng = np.random.default_rng(0)
    rgb = rng.integers(0, 256, size=(600, 800, 3), dtype=np.uint8)
    buf = io.BytesIO()
    Image.fromarray(rgb).save(buf, format="PNG")
    prep = VI.prepare(buf.getvalue())
    plan = prep.plan
    assert prep.patches.shape == (plan.vit_height * plan.vit_width, 588) and prep.patches.dtype == torch.bfloat16
    assert float(prep.patches.abs().max()) <= 1.0
    # patch (1, 2), channel 1, pixel (3, 4) is canvas pixel (17, 32) of the resized image
    im = np.asarray(Image.fromarray(rgb).resize((plan.resize_width, plan.resize_height), Image.BICUBIC))
    y, x = 14 + 3 - plan.top, 28 + 4 - plan.left
    want = ((im[y, x, 1] / 255.0) - 0.5) / 0.5
    got = float(prep.patches[1 * plan.vit_width + 2, 1 * 196 + 3 * 14 + 4])
    assert abs(got - want) < 0.01
    assert VI.identity(buf.getvalue()) == prep.identity != VI.identity(buf.getvalue(), "high")
    with pytest.raises(ValueError):
        VI.prepare(b"not an image")
    cache = VI.ImageCache(budget_bytes=3 * prep.patches.numel() * 2)
    for i in range(5):
        cache.put(bytes([i]), i, prep.patches.numel() * 2)
    assert cache.get(bytes([0])) is None and cache.get(bytes([4])) == 4 and cache.used <= cache.budget


@pytest.mark.gpu
def test_vision_tower_matches_oracle():
    from titanic_flash_41_b200.models import vision as V
    vc = VisionConfig(layers=2, hidden=256, heads=4, intermediate=384)
    d_model = 512
    W = V.init_vision_weights(vc, d_model, seed=1)
    gh, gw = 7, 10
    g = torch.Generator().manual_seed(2)
    patches = (torch.rand(gh * gw, 588, generator=g) * 2 - 1).bfloat16()
    want = V.VisionOracle(vc, d_model, W).encode(patches.float(), gh, gw)
    got = V.VisionTower(vc, d_model, W).encode(patches, gh, gw).float().cpu()
    assert got.shape == want.shape == (3 * (4 + 1) + 2, d_model)
    rel = float((got - want).norm() / want.norm())
    assert rel < 0.03, rel


def test_media_expansion_and_identity():
    import base64
    from PIL import Image
    from titanic_flash_41_b200.api import media as M
    buf = io.BytesIO()
    Image.fromarray(np.full((600, 600, 3), 200, dtype=np.uint8)).save(buf, format="PNG")
    uri = "data:image/png;base64," + base64.b64encode(buf.getvalue()).decode()
    cache = VI.ImageCache()
    pm = M.expand([5, 900, 6, 900, 7], [uri, uri], marker_id=900, image_token_id=901, cache=cache)
    n = pm.images[0].plan.tokens
    assert len(pm.tokens) == 3 + 2 * n and pm.tokens[1] == 901 and pm.offsets == [(1, n), (2 + n, n)]
    assert cache.hits == 1 and len(pm.identity) == 64
    assert M.expand([5], [], 900, 901).identity == ""
    for bad in ("http://example.com/x.png", "data:image/png;base64,@@@"):
        with pytest.raises(M.MediaError):
            M.expand([900], [bad], 900, 901)
    with pytest.raises(M.MediaError, match="disagree"):
        M.expand([5], [uri], 900, 901)


@pytest.mark.gpu
def test_prefill_with_image_span_embeddings():
    """Replacing embeddings through ``embeds`` with the tokens' own embeddings is a no-op; other rows change the logits."""
    from tests.test_engine_gpu import small_config
    from titanic_flash_41_b200.config import EngineConfig
    from titanic_flash_41_b200.models import engine as E, oracle
    from titanic_flash_41_b200.serve.prefill import run_prefill
    cfg = small_config()
    W = oracle.init_weights(cfg, 0)
    eng = E.Engine.from_weights(cfg, EngineConfig(reference_matmul=True, regions=2, max_context=512, prefill_widths=(64,)), W)
    p = torch.randint(0, cfg.vocab, (150,), generator=torch.Generator().manual_seed(1), dtype=torch.int32)
    base = run_prefill(eng, 0, p, 64)
    offs = torch.arange(70, 90)
    own = eng.embed_w[p[70:90].long().to(eng.dev)]
    same = run_prefill(eng, 1, p, 64, embeds=(offs, own))
    assert torch.equal(base, same)
    other = run_prefill(eng, 1, p, 64, embeds=(offs, own.flip(0)))
    assert not torch.equal(base, other) and torch.isfinite(other).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n,heads,spread", [(1, 1, 1.0), (127, 2, 1.0), (128, 1, 1.0), (129, 3, 4.0), (300, 2, 30.0), (1521, 16, 2.0)])
def test_dense_attention_kernel(n, heads, spread):
    """One key, a last tile of 1 / 127 / 128 keys, several tiles, and scores that grow along the keys so that the
    reference maximum moves (spread 30: by far more than the 2^8 it tolerates).

    Probabilities are rounded to bf16 (eight significant bits: at most 2^-8 relative) before PV and the output once
    more: |error| is at most 2^-8 (sum_k p_k |v_k| + |o|); the rest of the bound covers fp32 sums and the exponential."""
    from titanic_flash_41_b200.ops import native
    dev, n_pad = "cuda", -(-n // 128) * 128
    g = torch.Generator(device=dev).manual_seed(n)
    q, k, v = (torch.zeros(heads, n_pad, 64, dtype=torch.bfloat16, device=dev) for _ in range(3))
    ramp = torch.linspace(0.2, spread, n, device=dev)[None, :, None]
    q[:, :n] = torch.randn(heads, n, 64, generator=g, device=dev).bfloat16()
    k[:, :n] = (torch.randn(heads, n, 64, generator=g, device=dev) * ramp).bfloat16()
    v[:, :n] = torch.randn(heads, n, 64, generator=g, device=dev).bfloat16()
    out = torch.full((n + 1, heads * 64), 5.0, dtype=torch.bfloat16, device=dev)
    status = native.StatusWord(torch.device(dev))
    native.call("tf_vis_attention", q, k, v, out, n, n_pad, heads, heads * 64, 0.125, status.t)
    status.check()
    s = torch.einsum("hnd,hmd->hnm", q[:, :n].double(), k[:, :n].double()) * 0.125
    p = torch.softmax(s, -1)
    want = torch.einsum("hnm,hmd->nhd", p, v[:, :n].double())
    mag = torch.einsum("hnm,hmd->nhd", p, v[:, :n].double().abs())
    err = (out[:n].view(n, heads, 64).double() - want).abs()
    assert (err <= 2.0 ** -8 * 1.01 * (mag + want.abs()) + 1e-5).all(), float((err / (mag + want.abs())).max())
    assert (out[n] == 5.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n,width,off", [(3, 64, 1), (5, 72, 0), (5, 72, 3), (2, 1024, 5), (4, 77, 0), (1, 1, 0), (3, 1100, 1)])
def test_glue_kernels_on_and_off_the_vector_grain(n, width, off):
    """Eight elements an access, and the one-element form for widths off eight and for operands that start ``off`` elements
    behind a 16-byte boundary (a view into a larger tensor): stored values against fp64 of the same bf16 inputs.

    Sums and products of bf16 in fp32, one rounding to bf16 (2^-8 relative at most) each; an input that lies within fp32
    error of a rounding boundary may go either way, so that a chain of two roundings may differ by one more step."""
    from titanic_flash_41_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(width + off)

    def bf(*shape, fill=None):
        flat = torch.zeros(math.prod(shape) + off, dtype=torch.bfloat16, device="cuda")
        t = flat[off:].view(*shape)
        return t.copy_(torch.randn(*shape, generator=g, device="cuda") if fill is None else torch.full(shape, fill))

    def close(got, want, steps=1):
        return bool(((got.double() - want).abs() <= steps * 2.0 ** -8 * 1.01 * want.abs() + 1e-30).all())
    rnd = lambda t: t.bfloat16().double()
    x, delta, bias, w = bf(n, width), bf(n, width), bf(width), bf(width)
    d = lambda t: t.double()
    y = bf(n, width, fill=9.0)
    native.call("tf_vis_bias", x, bias, y, x.numel(), width)
    assert torch.equal(y, (x.float() + bias.float()).bfloat16())
    native.call("tf_vis_gelu", x, bias, y, x.numel(), width)
    v = rnd(x.float() + bias.float())
    assert bool(((d(y) - 0.5 * v * (1 + torch.erf(v * 0.5 ** 0.5))).abs() <= 2.0 ** -8 * 1.01 * d(y).abs() + 1e-6 * (1 + v.abs())).all())
    res = (x.float() + (delta.float() + bias.float()).bfloat16().float()).bfloat16()
    native.call("tf_vis_norm", x, delta, bias, w, y, n, width, 1e-6)
    assert torch.equal(x, res)
    assert close(y, d(res) * torch.rsqrt(d(res).pow(2).mean(-1, keepdim=True) + 1e-6) * d(w))
    gu = bf(n, 2 * width)
    native.call("tf_vis_swiglu", gu, y, n, width)
    assert close(y, rnd((d(gu[:, :width]) * torch.sigmoid(d(gu[:, :width]))).float()) * d(gu[:, width:]), steps=2)
    start, newline, end = bf(width), bf(width), bf(width)
    f, out = bf(2 * 3, width), bf(2 * 4 + 2, width, fill=9.0)
    native.call("tf_vis_span", f, bias, start, newline, end, out, 3, 10, width)
    fb = (f.float() + bias.float()).bfloat16()
    assert torch.equal(out, torch.cat([start[None], fb[:3], newline[None], fb[3:], newline[None], end[None]]))
    heads, n_pad = 2, n + 2
    qkv, qb = bf(n, 3 * heads * 64), bf(3 * heads * 64)
    q, k, vv = (bf(heads, n_pad, 64, fill=9.0) for _ in range(3))
    native.call("tf_vis_rope_split", qkv, qb, q, k, vv, n, n_pad, 2, heads)
    parts = (qkv.float() + qb.float()).bfloat16().view(n, 3, heads, 64)
    c = torch.arange(32, device="cuda")
    row = torch.arange(n, device="cuda")[:, None]
    ang = (torch.where(c < 16, row // 2, row % 2).double() * 10000.0 ** (-(c % 16).double() / 16))[:, None, :]
    for got, part in ((q, 0), (k, 1)):
        a, b = d(parts[:, part, :, :32]), d(parts[:, part, :, 32:])
        want = torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1).transpose(0, 1)
        assert bool(((d(got[:, :n]) - want).abs() <= 2.0 ** -8 * 1.01 * want.abs() + 1e-5).all()) and bool((got[:, n:] == 0).all())
    assert torch.equal(vv[:, :n], parts[:, 2].transpose(0, 1)) and bool((vv[:, n:] == 0).all())


@pytest.mark.gpu
def test_tower_with_weights_off_the_vector_grain():
    """Norm weights and biases on the device as views into one flat tensor (the tower keeps them as they are): the span
    follows the fp32 definition as with tensors of their own (the bound of the other tower test)."""
    from titanic_flash_41_b200.config import VisionConfig
    from titanic_flash_41_b200.models import vision as V
    vc, d_model, gh, gw = VisionConfig(layers=2, hidden=128, intermediate=256), 256, 8, 11
    W = {k: v.bfloat16().float() for k, v in V.init_vision_weights(vc, d_model, 3).items()}
    flat, at, dev = torch.zeros(sum(v.numel() + 1 for v in W.values()), dtype=torch.bfloat16, device="cuda"), 0, dict(W)
    for k, v in W.items():
        if v.dim() == 1:
            at += 1 if at % 2 == 0 else 2                   # an odd element: off the 16-byte (and the 4-byte) grain
            dev[k] = flat[at:at + v.numel()].copy_(v)
            at += v.numel()
    patches = (torch.rand(gh * gw, 588, generator=torch.Generator().manual_seed(1)) * 2 - 1).bfloat16()
    want = V.VisionOracle(vc, d_model, W).encode(patches.float(), gh, gw)
    tower = V.VisionTower(vc, d_model, dev)
    assert any(t.data_ptr() % 4 for t in tower.W.values())
    got = tower.encode(patches, gh, gw).float().cpu()
    assert float((got - want).norm() / want.norm()) < 0.03
