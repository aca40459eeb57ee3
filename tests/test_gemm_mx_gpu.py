"""Block-scaled tcgen05 GEMM (UE8M0 scales per 32 inputs applied by the tensor core) against fp32
PyTorch references of the same operands."""
import pytest
import torch

from titanic_flash_41_b200.models import engine as E
from titanic_flash_41_b200.ops import mx, native

pytestmark = pytest.mark.gpu
DEV = "cuda"
F8 = torch.float8_e4m3fn


def _rel(a, b):
    return float((a.float() - b.float()).norm() / (b.float().norm() + 1e-12))


def _mx_reference(x):
    """MXFP8 of rows: power-of-two scale per 32 inputs, smallest with amax / scale <= 448."""
    M, K = x.shape
    g = x.float().view(M, K // 32, 32)
    amax = g.abs().amax(-1)
    e = torch.ceil(torch.log2(amax.clamp_min(1e-38) / 448.0)).clamp(-127, 127)
    e = torch.where(amax > 0, e, torch.full_like(e, -127.0))
    q = (g * torch.exp2(-e)[:, :, None]).clamp(-448, 448).to(F8)
    return q.view(M, K), (e + 127).to(torch.uint8)


def _random_fp8(n, k, gen):
    b = torch.randint(0, 256, (n, k), device=DEV, dtype=torch.uint8, generator=gen)
    b[(b & 0x7F) == 0x7F] = 0x38                 # no NaN codes
    return b


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_quantiser_matches_the_mx_definition(dtype):
    torch.manual_seed(0)
    M, K = 70, 512
    x = (torch.randn(M, K, device=DEV) * torch.logspace(-3, 2, K, device=DEV)).to(dtype)
    x[3] = 0
    q = torch.zeros(M, K, dtype=torch.uint8, device=DEV)
    sf = mx.empty_units(M, K, 128, DEV)
    mx.quant_rows(x, M, K, q, sf)
    torch.cuda.synchronize()
    rq, rs = _mx_reference(x)
    assert torch.equal(mx.units_to_rowmajor(sf, M), rs)
    assert torch.equal(q.view(F8).float(), rq.float())


@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (300, 520, 512), (1000, 2048, 4096), (4200, 1024, 1024)])
def test_gemm_mx_fp8_weights(M, N, K):
    gen = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randn(M, K, device=DEV, generator=gen) * 2
    aq = torch.zeros(M, K, dtype=torch.uint8, device=DEV)
    sfa = mx.empty_units(M, K, 128, DEV)
    mx.quant_rows(x, M, K, aq, sfa)
    a_deq = aq.view(F8).float().view(M, K // 32, 32) * torch.exp2(mx.units_to_rowmajor(sfa, M).float() - 127)[:, :, None]
    bq = _random_fp8(N, K, gen)
    bs = torch.randint(118, 126, (N, K // 32), device=DEV, dtype=torch.uint8, generator=gen)
    sfb = mx.units_from_rowmajor(bs, K)
    b_deq = bq.view(F8).float().view(N, K // 32, 32) * torch.exp2(bs.float() - 127)[:, :, None]
    want = a_deq.view(M, K).double() @ b_deq.view(N, K).double().t()
    st = native.StatusWord(DEV)
    for dt, tol in ((torch.float32, 2e-5), (torch.bfloat16, 4e-3)):
        c = torch.full((M, N + 8), 7.0, device=DEV, dtype=dt)          # row pitch wider than N: the edge must stay untouched
        mx.gemm(aq, sfa, bq, sfb, c, M, N, K, st.t)
        torch.cuda.synchronize()
        st.check()
        assert _rel(c[:, :N], want) < tol
        assert bool((c[:, N:] == 7.0).all())


def test_gemm_mx_block_scales_of_dense_weights():
    """A dense FP8 matrix whose 128 x 128 scales are powers of two runs unchanged on the block-scaled
    path: same values as the fp32-scaled GEMM's operands."""
    torch.manual_seed(3)
    M, N, K = 256, 512, 1024
    w = torch.randn(N, K, device=DEV) * 0.05
    blk = w.view(N // 128, 128, K // 128, 128)
    s = torch.exp2(torch.ceil(torch.log2(blk.abs().amax(dim=(1, 3)) / 448.0)))
    wq = (blk / s[:, None, :, None]).clamp(-448, 448).to(F8).view(N, K)
    sfb = mx.units_from_block_scales(s.contiguous(), N, K)
    assert sfb is not None
    assert mx.units_from_block_scales((s * 1.5).contiguous(), N, K) is None
    x = torch.randn(M, K, device=DEV)
    aq = torch.zeros(M, K, dtype=torch.uint8, device=DEV)
    sfa = mx.empty_units(M, K, 128, DEV)
    mx.quant_rows(x, M, K, aq, sfa)
    a_deq = (aq.view(F8).float().view(M, K // 32, 32) * torch.exp2(mx.units_to_rowmajor(sfa, M).float() - 127)[:, :, None])
    w_deq = (wq.float().view(N // 128, 128, K // 128, 128) * s[:, None, :, None]).view(N, K)
    c = torch.zeros(M, N, device=DEV)
    st = native.StatusWord(DEV)
    mx.gemm(aq, sfa, wq.view(torch.uint8), sfb, c, M, N, K, st.t)
    torch.cuda.synchronize()
    st.check()
    assert _rel(c, a_deq.view(M, K).double() @ w_deq.double().t()) < 2e-5


def test_gemm_mx_grouped_mxfp4_experts():
    """Expert-sorted padded rows x packed e2m1 expert weights read as stored (no conversion pass)."""
    gen = torch.Generator(device=DEV).manual_seed(9)
    El, N, K = 3, 512, 1024
    tiles = torch.tensor([2, 0, 0, 1], dtype=torch.int32, device=DEV)        # expert of each 128-row tile
    ntile = torch.tensor([4], dtype=torch.int32, device=DEV)
    cap = 6 * 128                                                            # two tiles beyond num_m_tiles stay untouched
    x = torch.randn(cap, K, device=DEV, generator=gen)
    aq = torch.zeros(cap, K, dtype=torch.uint8, device=DEV)
    sfa = mx.empty_units(cap, K, 128, DEV)
    mx.quant_rows(x, cap, K, aq, sfa)
    a_deq = (aq.view(F8).float().view(cap, K // 32, 32) * torch.exp2(mx.units_to_rowmajor(sfa, cap).float() - 127)[:, :, None])
    pk = torch.randint(0, 256, (El, N, K // 2), device=DEV, dtype=torch.uint8, generator=gen)
    sc = torch.randint(118, 126, (El, N, K // 32), device=DEV, dtype=torch.uint8, generator=gen)
    w = E.dequant_mxfp4(pk, sc)                                              # [El, N, K]
    sfb = mx.units_from_rowmajor(sc, K)
    c = torch.full((cap, N), 5.0, device=DEV, dtype=torch.bfloat16)
    st = native.StatusWord(DEV)
    mx.gemm(aq, sfa, pk, sfb, c, cap, N, K, st.t, b_fp4=True, b_rows=El * N, tile_expert=tiles, num_m_tiles=ntile)
    torch.cuda.synchronize()
    st.check()
    for i, e in enumerate(tiles.tolist()):
        rows = slice(i * 128, (i + 1) * 128)
        assert _rel(c[rows], a_deq.view(cap, K)[rows].double() @ w[e].double().t()) < 4e-3
    assert bool((c[4 * 128:] == 5.0).all())


def test_gemm_mx_refuses_bad_arguments():
    st = native.StatusWord(DEV)
    a = torch.zeros(128, 128, dtype=torch.uint8, device=DEV)
    sf = mx.empty_units(128, 128, 128, DEV)
    sfb = mx.empty_units(256, 128, 256, DEV)
    c = torch.zeros(128, 256, device=DEV)
    with pytest.raises(native.NativeError):
        native.call("tf_gemm_mx", a, 128, a, 128, 256, 0, sf, sf.shape[1], sfb, sfb.shape[1], c, 256, 0, 128, 256, 96, None,
                    None, st.t)                                            # K not a multiple of 128
    with pytest.raises(native.NativeError):
        native.call("tf_gemm_mx", a, 128, a, 128, 256, 0, sf, 1, sfb, sfb.shape[1], c, 256, 0, 128, 256, 128, None, None,
                    st.t)                                                  # too few scale units for the rows


@pytest.mark.gpu
@pytest.mark.parametrize("rows,K,off", [(1, 128, 0), (127, 4096, 0), (129, 4224, 0), (640, 8320, 0), (130, 256, 1), (131, 4096, 4),
                                        (261, 8192, 0), (258, 2048, 0), (1025, 5120, 0)])
def test_scale_units_transpose(rows, K, off):
    """Both forms (16-byte pieces for 32, 16 or 8 words a row piece; words) with ragged edges, and sources off the 16-byte
    and the 4-byte boundary: bytes move unchanged."""
    from titanic_flash_41_b200.ops import mx, native
    g = torch.Generator(device="cuda").manual_seed(rows)
    flat = torch.randint(0, 256, (rows * (K // 32) + off,), generator=g, device="cuda", dtype=torch.uint8)
    s = flat[off:].view(rows, K // 32)
    out = torch.full((K // 128, mx.sf_units(rows, 256), 128), 7, dtype=torch.uint8, device="cuda")
    native.call("tf_mx_sf_to_units", s, out, rows, K, out.shape[1])
    assert torch.equal(mx.units_to_rowmajor(out, rows), s)
    pad = out.view(K // 128, -1, 4)[:, rows:]
    assert int((pad != 7).sum()) == 0                      # rows beyond the matrix are left alone


@pytest.mark.parametrize("El,e_lo,pairs", [(1, 0, 5), (33, 7, 700), (512, 0, 3000), (700, 64, 20000)])
def test_moe_plan_tables(El, e_lo, pairs):
    """Experts below, at and beyond one pass of the offset scan, experts without rows and pairs of other ranks: padded offsets,
    tile table, placement; and the counters are ready for the next call."""
    g = torch.Generator().manual_seed(El)
    ids = torch.randint(0, e_lo + El + 40, (pairs,), generator=g, dtype=torch.int32)
    ids[ids % 5 == 1] = e_lo                                   # one expert over several tiles, others empty
    i32 = lambda n: torch.full((n,), -5, dtype=torch.int32, device=DEV)
    counts = torch.zeros(El, dtype=torch.int32, device=DEV)
    cap = pairs // 128 + El + 1
    for _ in range(2):
        offs, cur, tile_e, nt, pad, dst = i32(El + 1), i32(El), i32(cap), i32(1), i32(1), i32(pairs)
        tile_r = i32(cap)
        native.call("tf_moe_plan_rows", ids.to(DEV), pairs, e_lo, El, counts, offs, cur, tile_e, tile_r, cap, nt, pad, dst)
        local = ids.long() - e_lo
        mine = (local >= 0) & (local < El)
        cnt = torch.bincount(local[mine], minlength=El)
        tiles = (cnt + 127) // 128
        want = torch.cat([torch.zeros(1, dtype=torch.long), torch.cumsum(tiles * 128, 0)])
        assert torch.equal(offs.cpu().long(), want) and int(nt) == int(tiles.sum()) and int(pad) == int(want[-1])
        assert torch.equal(tile_e[:int(nt)].cpu().long(), torch.arange(El).repeat_interleave(tiles))
        first = torch.cat([torch.arange(int(t)) for t in tiles]) if int(nt) else torch.zeros(0)
        assert torch.equal(tile_r[:int(nt)].cpu().long(), (cnt.repeat_interleave(tiles) - 128 * first).clamp(max=128).long())
        d = dst.cpu().long()
        assert bool((d[~mine] == -1).all()) and d[mine].unique().numel() == int(mine.sum())
        assert bool(((d[mine] >= want[local[mine]]) & (d[mine] < want[local[mine]] + cnt[local[mine]])).all())
        assert int(counts.abs().sum()) == 0


def test_grouped_gemm_and_swiglu_store_only_rows_that_count():
    """Tiles of 1, 32, 33, 127 and 128 rows: rows that count equal the form that stores whole tiles bit for bit, padding keeps
    what it held; the activation kernel skips the same rows."""
    gen = torch.Generator(device=DEV).manual_seed(5)
    rows = torch.tensor([1, 32, 33, 127, 128], dtype=torch.int32, device=DEV)
    El, N, K, M = 5, 256, 256, 640
    a = _random_fp8(M, K, gen)
    sfa, sfb = torch.full((K // 128, M // 32, 128), 127, dtype=torch.uint8, device=DEV), torch.full((K // 128, El * N // 32, 128), 124, dtype=torch.uint8, device=DEV)
    w = torch.randint(0, 256, (El * N, K // 2), dtype=torch.uint8, device=DEV, generator=gen)
    tiles, nt = torch.arange(5, dtype=torch.int32, device=DEV), torch.tensor([5], dtype=torch.int32, device=DEV)
    st = native.StatusWord(DEV)
    whole, part = torch.zeros(M, N, device=DEV), torch.full((M, N), 3.0, device=DEV)
    kw = dict(b_fp4=True, b_rows=El * N, tile_expert=tiles, num_m_tiles=nt)
    mx.gemm(a, sfa, w, sfb, whole, M, N, K, st.t, **kw)
    mx.gemm(a, sfa, w, sfb, part, M, N, K, st.t, tile_rows=rows, **kw)
    st.check()
    live = (torch.arange(M, device=DEV) % 128) < rows.repeat_interleave(128)
    assert torch.equal(part[live], whole[live]) and bool((part[~live] == 3.0).all())
    y = torch.randn(M, 2 * N, device=DEV, generator=gen).bfloat16()
    q = [torch.full((M, N), 9, dtype=torch.uint8, device=DEV) for _ in range(2)]
    sf = [torch.full((N // 128, M // 32, 128), 9, dtype=torch.uint8, device=DEV) for _ in range(2)]
    n = torch.tensor([M], dtype=torch.int32, device=DEV)
    for i, tr in enumerate((None, rows)):
        native.call("tf_swiglu_rows_mx_units", y, 2 * N, q[i], sf[i], M // 32, M, N, 10.0, n, tr)
    assert torch.equal(q[1][live], q[0][live]) and bool((q[1][~live] == 9).all())
    assert torch.equal(mx.units_to_rowmajor(sf[1], M)[live], mx.units_to_rowmajor(sf[0], M)[live])


@pytest.mark.parametrize("M,N,K", [(1, 136, 128), (33, 128, 256), (197, 9864, 512), (255, 384, 896), (257, 512, 1152), (1500, 4096, 640)])
def test_gemm_mx_dense_tiles(M, N, K):
    """Row tiles of every width the tile rule takes, a last tile of a few rows, feature blocks that end inside a CTA's 128
    features or in the pair's second CTA: the same operands in fp64.  fp32 accumulation of K exact products: 2e-5 as above."""
    gen = torch.Generator(device=DEV).manual_seed(M + K)
    aq, bq = _random_fp8(M, K, gen), _random_fp8(N, K, gen)
    sa = torch.randint(118, 126, (M, K // 32), device=DEV, dtype=torch.uint8, generator=gen)
    sb = torch.randint(118, 126, (N, K // 32), device=DEV, dtype=torch.uint8, generator=gen)
    deq = lambda q, s: (q.view(F8).double().view(-1, K // 32, 32) * torch.exp2(s.double() - 127)[:, :, None]).view(-1, K)
    want = deq(aq, sa) @ deq(bq, sb).t()
    st = native.StatusWord(DEV)
    for dt, tol in ((torch.float32, 2e-5), (torch.bfloat16, 4e-3)):
        c = torch.full((M + 1, N + 8), 7.0, device=DEV, dtype=dt)
        mx.gemm(aq, mx.units_from_rowmajor(sa, K, 128), bq, mx.units_from_rowmajor(sb, K), c, M, N, K, st.t)
        st.check()
        assert _rel(c[:M, :N], want) < tol
        assert bool((c[:, N:] == 7.0).all()) and bool((c[M] == 7.0).all())


@pytest.mark.parametrize("K,tile_max,two", [(512, 32, True), (768, 96, True), (1280, 160, False), (1024, 192, True), (2304, 256, False)])
def test_gemm_mx_experts_tiles(K, tile_max, two):
    """Experts of 0, 1, 31, 33, tile_max and more rows through the tile plan, scales row-major as stored (rows of a multiple
    of 16 bytes and of 8 bytes off it), one and two matrices: live rows against fp64, padding keeps what it held."""
    gen = torch.Generator(device=DEV).manual_seed(K)
    counts = [1, 31, 0, 33, tile_max, tile_max + 1, 300]
    El, N, n = len(counts), 256, sum(counts)
    ids = torch.repeat_interleave(torch.arange(El), torch.tensor(counts))[torch.randperm(n)].int().to(DEV)
    i32 = lambda k: torch.full((k,), -5, dtype=torch.int32, device=DEV)
    cap, room = -(-(n + El * 31) // 32) * 32, n // tile_max + El
    offs, cur, te, r0, tr, nt, pad, dst = i32(El + 1), i32(El), i32(room), i32(room), i32(room), i32(1), i32(1), i32(n)
    native.call("tf_moe_plan_tiles", ids, n, 0, El, torch.zeros(El, dtype=torch.int32, device=DEV), offs, cur, te, r0, tr, tile_max,
                room, nt, pad, dst)
    want_offs = [0]
    for c in counts:
        want_offs.append(want_offs[-1] + -(-c // 32) * 32)
    assert offs.tolist() == want_offs and int(pad) == want_offs[-1] <= cap
    seen = []
    for t in range(int(nt)):
        e, a, m = int(te[t]), int(r0[t]), int(tr[t])
        assert a % 32 == 0 and 0 < m <= tile_max
        seen += list(range(a, a + m))
    assert sorted(dst.tolist()) == sorted(seen) and len(set(seen)) == n
    aq = _random_fp8(cap, K, gen)
    sa = torch.randint(118, 126, (cap, K // 32), device=DEV, dtype=torch.uint8, generator=gen)
    pk = [torch.randint(0, 256, (El, N, K // 2), device=DEV, dtype=torch.uint8, generator=gen) for _ in range(2)]
    sc = [torch.randint(118, 126, (El, N, K // 32), device=DEV, dtype=torch.uint8, generator=gen) for _ in range(2)]
    a = (aq.view(F8).double().view(cap, K // 32, 32) * torch.exp2(sa.double() - 127)[:, :, None]).view(cap, K)
    st = native.StatusWord(DEV)
    for dt, tol in ((torch.float32, 2e-5), (torch.bfloat16, 4e-3)):
        c = torch.full((cap, 2 * N + 8), 5.0, device=DEV, dtype=dt)
        mx.gemm_experts(aq, mx.units_from_rowmajor(sa, K, 128), pk[0], pk[1] if two else None, sc[0], sc[1] if two else None, El * N,
                        c, cap, N, K, (te, r0, tr, nt, tile_max, room), st.t)
        st.check()
        expert = torch.full((cap,), -1, device=DEV)
        expert[dst.long()] = ids.long()
        for e in range(El):
            rows = expert == e
            for j in range(2 if two else 1):
                if int(rows.sum()):
                    w = E.dequant_mxfp4(pk[j][e], sc[j][e]).double()
                    assert _rel(c[rows, j * N:(j + 1) * N], a[rows] @ w.t()) < tol
        assert bool((c[expert < 0] == 5.0).all()) and bool((c[:, (2 if two else 1) * N:] == 5.0).all())


@pytest.mark.parametrize("M", [1, 130, 200, 256])
def test_grouped_gemm_stores_no_row_behind_the_last_and_none_of_an_empty_tile(M):
    """Grouped rows that end inside a 128-row tile, with and without the rows of each tile, an empty tile among them, and a
    count of tiles beyond the list: C keeps what it held behind row M and in every row that does not count."""
    gen = torch.Generator(device=DEV).manual_seed(M)
    El, N, K, tiles = 2, 256, 256, -(-M // 128)
    a = _random_fp8(M, K, gen)
    sfa = torch.full((K // 128, tiles * 4, 128), 127, dtype=torch.uint8, device=DEV)
    sfb = torch.full((K // 128, El * N // 32, 128), 124, dtype=torch.uint8, device=DEV)
    w = torch.randint(0, 256, (El * N, K // 2), dtype=torch.uint8, device=DEV, generator=gen)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    te, st = i32([1, 0][:tiles]), native.StatusWord(DEV)
    full = a.view(F8).double() @ E.dequant_mxfp4(w.view(El, N, K // 2), torch.full((El, N, K // 32), 124, dtype=torch.uint8, device=DEV)).double().transpose(1, 2)
    for rows in (None, [0, 128], [128, 0], [1, 77]):
        for dt, tol in ((torch.float32, 2e-5), (torch.bfloat16, 4e-3)):
            c = torch.full((M + 256, N), 3.0, device=DEV, dtype=dt)
            mx.gemm(a, sfa, w, sfb, c, M, N, K, st.t, b_fp4=True, b_rows=El * N, tile_expert=te, num_m_tiles=i32([tiles + (rows is not None)]),
                    tile_rows=None if rows is None else i32(rows[:tiles]))
            st.check()
            live = torch.zeros(M + 256, dtype=torch.bool, device=DEV)
            for t in range(tiles):
                n = min(128 if rows is None else rows[t], M - 128 * t)
                live[128 * t:128 * t + n] = True
                if n > 0:
                    assert _rel(c[128 * t:128 * t + n], full[int(te[t])][128 * t:128 * t + n]) < tol
            assert bool((c[~live] == 3.0).all())
