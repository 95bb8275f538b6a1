"""Quantised-weight tcgen05 GEMM (weights expanded in flight) against torch fp32 matmul of the same dequantised
weights and bf16 activations."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _status():
    return torch.zeros(1, dtype=torch.int32, device=DEV)


def _weight(t, shape, K, seed):
    from bloomery_b200.formats.resident import quantize_resident, resident_type
    from bloomery_b200.ops.decode import QWeight
    g = torch.Generator().manual_seed(seed)
    rows = 1
    for d in shape:
        rows *= d
    w = torch.randn(rows, K, generator=g) * 0.05
    res, ref = quantize_resident(w, t)
    return QWeight(res.to(DEV).reshape(*shape, -1).contiguous(), resident_type(t), K), ref.reshape(*shape, K).to(DEV)


@pytest.mark.parametrize("t", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "FP8_B128", "NVFP4", "IQ4_NL"])
@pytest.mark.parametrize("rows,tile", [(300, 128), (45, 32), (128, 128), (64, 64), (100, 64)])
def test_dense_qgemm(t, rows, tile):
    from bloomery_b200.ops import gemm as G
    N, K = 200, 1024                                            # N not a multiple of 128: the last weight tile is ragged
    qw, ref_w = _weight(t, (N,), K, 1)
    torch.manual_seed(2)
    X = (torch.randn(rows, K, device=DEV) * 0.5).bfloat16()
    R = torch.randn(rows, N, device=DEV)
    C = torch.full((rows, N), float("nan"), device=DEV)
    st = _status()
    tiles = G.TileTable.dense(rows, DEV, tile)
    G.qgemm(X, qw, tiles, out_f32=C, resid=R, status=st)
    torch.cuda.synchronize()
    assert int(st) == 0
    ref = X.float() @ ref_w.bfloat16().float().T + R
    # tiles below 128 tokens use the short expander (scale and offset of a block rounded to bf16 before the FMA)
    # (NVFP4 rounds its group scale to bf16 there)
    tol = dict(rtol=1e-3, atol=1e-2) if tile == 128 else dict(rtol=1e-2, atol=3e-2)
    assert torch.allclose(C, ref, **tol), (C - ref).abs().max()
    C2 = torch.zeros_like(C)
    G.qgemm(X, qw, tiles, out_f32=C2, resid=R, status=st)
    assert torch.equal(C, C2)                                   # bit-identical rerun


@pytest.mark.parametrize("t", ["Q8_0", "FP8_B128", "NVFP4", "IQ4_NL"])
@pytest.mark.parametrize("tile", [32, 64, 128])
def test_the_exact_form_multiplies_the_weights_of_the_bf16_copies(t, tile):
    """Rows of the identity read every weight out of the product as it was multiplied: the fp32 value rounded to bf16
    once, bit for bit what the bf16 copies hold; the SwiGLU pair too."""
    from bloomery_b200.ops import gemm as G
    N, K = 136, 512
    (w, _), (w2, _) = _weight(t, (N,), K, 21), _weight(t, (N,), K, 22)
    copies = [torch.zeros(N, K, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    for q, c in zip((w, w2), copies):
        G.dequant_bf16(q, c)
    X = torch.eye(K, dtype=torch.bfloat16, device=DEV)
    st, tiles = _status(), G.TileTable.dense(K, DEV, tile)
    C, D = (torch.full((K, N), float("nan"), device=DEV) for _ in range(2))
    G.qgemm(X, w, tiles, out_f32=C, status=st, exact=True)
    G.qgemm(X, w, tiles, out_f32=D, W2=w2, status=st, exact=True)
    torch.cuda.synchronize()
    assert int(st) == 0
    g, u = (c.float().T for c in copies)
    assert torch.equal(C, g)
    # fp32 exponential and division: a few 2^-22
    assert torch.allclose(D, torch.nn.functional.silu(g) * u, rtol=4e-6, atol=1e-12)


@pytest.mark.parametrize("t", ["Q4_K", "Q5_K", "Q6_K", "Q8_0", "FP8_B128", "NVFP4", "IQ4_NL"])
@pytest.mark.parametrize("tile,K", [(32, 256), (32, 2304), (64, 256), (64, 2304)])
def test_the_split_form_keeps_sixteen_bits_of_every_weight(t, tile, K):
    """Identity rows again: value and remainder add up to the fp32 weight to 2^-17 of it; depths of one super-block and of
    several turns of the operand ring, the SwiGLU pair and a depth shared by several CTAs too."""
    from bloomery_b200.ops import gemm as G
    N = 136
    (w, v), (w2, v2) = _weight(t, (N,), K, 23), _weight(t, (N,), K, 24)
    X = torch.eye(K, dtype=torch.bfloat16, device=DEV)[:97 if K > 256 else K].contiguous()
    X[5, K - 1] = 1                                              # a row that reaches both ends of the depth
    st, tiles = _status(), G.TileTable.dense(X.shape[0], DEV, tile)
    C, S, D = (torch.full((X.shape[0], N), float("nan"), device=DEV) for _ in range(3))
    G.qgemm(X, w, tiles, out_f32=C, status=st, fine=True)
    G.qgemm(X, w, tiles, out_f32=S, status=st, fine=True, work=G.QgemmWork(DEV))
    if tile == 32:
        G.qgemm(X, w, tiles, out_f32=D, W2=w2, status=st, fine=True)
    torch.cuda.synchronize()
    assert int(st) == 0
    g, u = (X.float() @ m.T for m in (v, v2))
    # what the remainder's own rounding leaves is 2^-18 of a weight; row 5 adds two weights
    bound = 2 ** -17 * (X.float() @ v.abs().T)
    assert bool(((C - g).abs() <= bound).all()), (C - g).abs().max()
    assert bool(((S - g).abs() <= bound).all())
    if tile == 32:
        # the slope of silu is below 1.1; its fp32 exponential and division add a few 2^-22
        silu = torch.nn.functional.silu(g)
        bound2 = 1.1 * u.abs() * bound + silu.abs() * 2 ** -17 * (X.float() @ v2.abs().T) + 4e-6 * (silu * u).abs()
        assert bool(((D - silu * u).abs() <= bound2).all()), (D - silu * u).abs().max()


@pytest.mark.parametrize("gt,dt", [("Q4_K", "Q6_K"), ("FP8_B128", "FP8_B128"), ("NVFP4", "NVFP4")])
@pytest.mark.parametrize("tile,T", [(128, 700), (32, 24)])
def test_grouped_dual_swiglu_and_scatter_quantised(tile, T, gt, dt):
    """The MoE path on quantised experts: rows grouped by expert, gate/up fused with SwiGLU (Q4_K), down (Q6_K)
    scattered with the router weights; prompt-sized tiles and decode-batch tiles."""
    from bloomery_b200.ops import gemm as G
    torch.manual_seed(3)
    E, k, H, I_ = 8, 2, 512, 256
    wg, ref_g = _weight(gt, (E, I_), H, 4)
    wu, ref_u = _weight(gt, (E, I_), H, 5)
    wd, ref_d = _weight(dt, (E, H), I_, 6)
    ids = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).to(torch.int32).to(DEV)
    ids[5, 1] = -1
    wts = torch.rand(T, k, device=DEV)
    x = (torch.randn(T, H, device=DEV) * 0.5).bfloat16()
    n = T * k
    cap = n + 128
    pos_of = torch.zeros(n, dtype=torch.int32, device=DEV)
    dst_row = torch.zeros(cap, dtype=torch.int32, device=DEV)
    row_scale = torch.zeros(cap, device=DEV)
    tiles = G.TileTable(n, E, DEV, tile)
    G.moe_plan(ids, wts, E, tiles, pos_of, dst_row, row_scale)
    Ap = torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV)
    G.gather_rows_bf16(x, dst_row, tiles.offsets[E:E + 1], cap, k, Ap)
    act = torch.zeros(cap, I_, dtype=torch.bfloat16, device=DEV)
    st = _status()
    G.qgemm(Ap, wg, tiles, out_bf16=act, W2=wu, status=st)
    slot_out = torch.zeros(n, H, device=DEV)
    G.qgemm(act, wd, tiles, out_f32=slot_out, dst_row=dst_row, row_scale=row_scale, status=st)
    resid = torch.randn(T, H, device=DEV)
    y = torch.zeros(T, H, device=DEV)
    G.moe_combine(slot_out, pos_of, T, k, resid, y)
    torch.cuda.synchronize()
    assert int(st) == 0
    ref = resid.clone()
    xf = x.float()
    Wg, Wu, Wd = ref_g.bfloat16().float(), ref_u.bfloat16().float(), ref_d.bfloat16().float()
    for t_ in range(T):
        for j in range(k):
            e = int(ids[t_, j])
            if e < 0:
                continue
            a = (torch.nn.functional.silu(xf[t_] @ Wg[e].T) * (xf[t_] @ Wu[e].T)).bfloat16().float()
            ref[t_] += wts[t_, j] * (a @ Wd[e].T)
    assert torch.allclose(y, ref, rtol=2e-2, atol=2e-2), (y - ref).abs().max()


def _fp8_acts(X):
    """Device quantisation of bf16 rows and the fp32 values the codes stand for."""
    from bloomery_b200.formats.planes import e4m3_decode
    from bloomery_b200.ops import gemm as G
    rows, K = X.shape
    codes = torch.zeros(rows, K, dtype=torch.uint8, device=DEV)
    scales = torch.zeros(rows, K // 128, device=DEV)
    G.fp8_rows(X, codes, scales)
    vals = e4m3_decode(codes.cpu()).to(DEV).reshape(rows, K // 128, 128) * scales[:, :, None]
    return codes, scales, vals.reshape(rows, K)


def test_fp8_rows_quantise_within_half_a_step_and_fuse_the_norm():
    from bloomery_b200.ops import gemm as G
    torch.manual_seed(11)
    X = (torch.randn(37, 1024, device=DEV) * torch.rand(37, 1, device=DEV) * 3).bfloat16()
    X[3, 128:256] = 0                                            # an all-zero block keeps scale 1 and codes 0
    codes, scales, vals = _fp8_acts(X)
    amax = X.float().reshape(37, 8, 128).abs().amax(-1)
    assert torch.allclose(scales, torch.where(amax > 0, amax / 448, torch.ones_like(amax)), rtol=1e-6)
    err = (vals - X.float()).abs().reshape(37, 8, 128)
    # E4M3 keeps 3 mantissa bits: half a step is 1/16 of the value's power of two, at most 1/16 of the block maximum
    assert bool((err <= amax[:, :, None] / 16 * 1.001 + 1e-12).all())
    assert int(codes[3, 128:256].max()) == 0
    xf = torch.randn(5, 512, device=DEV)
    gain = torch.rand(512, device=DEV) + 0.5
    c2 = torch.zeros(5, 512, dtype=torch.uint8, device=DEV)
    s2 = torch.zeros(5, 4, device=DEV)
    G.fp8_rows(xf, c2, s2, gain=gain, eps=1e-6)
    normed = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6) * gain
    assert torch.allclose(s2, normed.reshape(5, 4, 128).abs().amax(-1) / 448, rtol=1e-4)


@pytest.mark.parametrize("rows", [45, 32, 7])
def test_fp8_block_scaled_dense_gemm(rows):
    from bloomery_b200.ops import gemm as G
    N, K = 200, 1024                                            # N not a multiple of 128: the last weight tile is ragged
    qw, ref_w = _weight("FP8_B128", (N,), K, 1)
    torch.manual_seed(2)
    X = (torch.randn(rows, K, device=DEV) * 0.5).bfloat16()
    codes, scales, xv = _fp8_acts(X)
    R = torch.randn(rows, N, device=DEV)
    C = torch.full((rows, N), float("nan"), device=DEV)
    st = _status()
    tiles = G.TileTable.dense(rows, DEV, 32)
    G.fp8_gemm(codes, scales, qw, tiles, out_f32=C, resid=R, status=st)
    torch.cuda.synchronize()
    assert int(st) == 0
    ref = xv.double() @ ref_w.double().T + R.double()            # the quantised operands' own values, exact products
    assert torch.allclose(C.double(), ref, rtol=1e-4, atol=1e-4), (C.double() - ref).abs().max()
    C2 = torch.zeros_like(C)
    G.fp8_gemm(codes, scales, qw, tiles, out_f32=C2, resid=R, status=st)
    assert torch.equal(C, C2)
    plain = X.float() @ ref_w.T + R                               # and the activation rounding stays a small error
    assert float((C - plain).abs().max()) < 0.05 * float(plain.abs().max())


@pytest.mark.parametrize("rows,N,K,dual", [(1, 200, 128, False), (5, 38400, 256, False), (9, 38400, 128, True),
                                           (33, 19200, 640, False), (29, 38400, 256, True), (4768, 128, 73728, False)])
def test_fp8_tiles_of_one_block_follow_each_other(rows, N, K, dual):
    """More tiles than blocks, so scales and routing come in a tile ahead: few, ragged and full token groups, a row of
    scales that ends inside a load, and a K whose scales fit shared memory only once."""
    from bloomery_b200.ops import gemm as G
    qw, ref_w = _weight("FP8_B128", (N,), K, 1)
    qw2, ref_w2 = _weight("FP8_B128", (N,), K, 2) if dual else (None, None)
    torch.manual_seed(3)
    X = (torch.randn(rows, K, device=DEV) * 0.5).bfloat16()
    codes, scales, xv = _fp8_acts(X)
    dst = torch.randperm(rows, device=DEV).to(torch.int32)
    factor = torch.rand(rows, device=DEV) + 0.5
    C = torch.full((rows + 1, N), float("nan"), device=DEV)
    st = _status()
    G.fp8_gemm(codes, scales, qw, G.TileTable.dense(rows, DEV, 32), out_f32=C, W2=qw2, dst_row=dst, row_scale=factor, status=st)
    torch.cuda.synchronize()
    assert int(st) == 0 and bool(C[rows].isnan().all())
    pick = torch.arange(rows, device=DEV) if rows < 64 else torch.cat([torch.arange(0, rows, 97, device=DEV), torch.tensor([rows - 1], device=DEV)])
    # an instruction of 32 values rounds (or cuts) once, the promotion of a block twice, each at most 2^-23 of the terms' sum
    step = (K / 32 + 2 * K / 128 + 2) * 2.0 ** -23
    x = xv[pick].double()
    ref, tol = x @ ref_w.double().T, step * (x.abs() @ ref_w.double().abs().T)
    if dual:
        up, tol_up = x @ ref_w2.double().T, step * (x.abs() @ ref_w2.double().abs().T)
        gate = torch.nn.functional.silu(ref)                     # slope at most 1.1; the exponential and the division a few units
        tol = 1.1 * tol * (up.abs() + tol_up) + gate.abs() * tol_up + 2.0 ** -18 * (gate * up).abs()
        ref = gate * up
    f = factor[pick].double()[:, None]
    err = (C[dst[pick].long()].double() - ref * f).abs()
    assert bool((err <= (tol * f + 2.0 ** -22 * (ref * f).abs() + 1e-30)).all()), (err - tol * f).max()


def test_fp8_block_scaled_grouped_dual_and_scatter():
    from bloomery_b200.ops import gemm as G
    torch.manual_seed(3)
    E, k, H, I_, T = 8, 2, 512, 256, 24
    wg, ref_g = _weight("FP8_B128", (E, I_), H, 4)
    wu, ref_u = _weight("FP8_B128", (E, I_), H, 5)
    wd, ref_d = _weight("FP8_B128", (E, H), I_, 6)
    ids = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).to(torch.int32).to(DEV)
    ids[5, 1] = -1
    wts = torch.rand(T, k, device=DEV)
    x = (torch.randn(T, H, device=DEV) * 0.5).bfloat16()
    n = T * k
    cap = n + 128
    pos_of = torch.zeros(n, dtype=torch.int32, device=DEV)
    dst_row = torch.zeros(cap, dtype=torch.int32, device=DEV)
    row_scale = torch.zeros(cap, device=DEV)
    tiles = G.TileTable(n, E, DEV, 32)
    G.moe_plan(ids, wts, E, tiles, pos_of, dst_row, row_scale)
    Ap = torch.zeros(cap, H, dtype=torch.bfloat16, device=DEV)
    G.gather_rows_bf16(x, dst_row, tiles.offsets[E:E + 1], cap, k, Ap)
    ac, asc, _ = _fp8_acts(Ap)
    act = torch.zeros(cap, I_, dtype=torch.bfloat16, device=DEV)
    st = _status()
    G.fp8_gemm(ac, asc, wg, tiles, out_bf16=act, W2=wu, status=st)
    bc, bsc, _ = _fp8_acts(act)
    slot_out = torch.zeros(n, H, device=DEV)
    G.fp8_gemm(bc, bsc, wd, tiles, out_f32=slot_out, dst_row=dst_row, row_scale=row_scale, status=st)
    resid = torch.randn(T, H, device=DEV)
    y = torch.zeros(T, H, device=DEV)
    G.moe_combine(slot_out, pos_of, T, k, resid, y)
    torch.cuda.synchronize()
    assert int(st) == 0
    ref = resid.clone()
    xf = x.float()
    for t_ in range(T):
        for j in range(k):
            e = int(ids[t_, j])
            if e < 0:
                continue
            a = torch.nn.functional.silu(xf[t_] @ ref_g[e].T) * (xf[t_] @ ref_u[e].T)
            ref[t_] += wts[t_, j] * (a @ ref_d[e].T)
    # activations rounded to E4M3 twice (in front of gate / up and in front of down): a few percent of the expert sum
    assert float((y - ref).abs().max()) < 0.06 * float((ref - resid).abs().max()) + 1e-3, (y - ref).abs().max()


@pytest.mark.parametrize("t", ["Q4_K", "Q6_K", "NVFP4"])
@pytest.mark.parametrize("rows,tile,N,K", [(5, 32, 512, 1024), (33, 32, 128, 4096), (64, 64, 2048, 4096), (17, 64, 200, 768)])
def test_dense_qgemm_with_its_depth_split(t, rows, tile, N, K):
    """A product of few tiles shares each tile's depth among CTAs: the same sums to fp32 rounding, the same bits on every
    run, and tickets that are ready for the next launch."""
    from bloomery_b200.ops import gemm as G
    from bloomery_b200.ops.decode import sm_count
    qw, _ = _weight(t, (N,), K, 1)
    torch.manual_seed(2)
    X = (torch.randn(rows, K, device=DEV) * 0.5).bfloat16()
    R = torch.randn(rows, N, device=DEV)
    tiles = G.TileTable.dense(rows, DEV, tile)
    assert G.qgemm_splits(tiles.fixed * ((N + 127) // 128), K // 256, sm_count()) > 1
    st, work = _status(), G.QgemmWork(DEV)
    C = [torch.full((rows, N), float("nan"), device=DEV) for _ in range(3)]
    G.qgemm(X, qw, tiles, out_f32=C[0], resid=R, status=st)
    for c in C[1:]:
        G.qgemm(X, qw, tiles, out_f32=c, resid=R, status=st, work=work)
    torch.cuda.synchronize()
    assert int(st) == 0 and int(work.tickets.abs().max()) == 0
    assert torch.equal(C[1], C[2])
    # K products of order 0.5 x 0.05, their fp32 sums regrouped once: sqrt(K) * 0.025 * 2^-24 * a few, far below 1e-4
    assert torch.allclose(C[0], C[1], rtol=1e-5, atol=1e-4), (C[0] - C[1]).abs().max()


def test_the_split_takes_equal_shares_and_no_more_ctas_than_processors():
    from bloomery_b200.ops import gemm as G
    for tiles in (1, 4, 16, 32, 147, 148, 1187):
        for blocks in (1, 2, 3, 8, 16, 30):
            s = G.qgemm_splits(tiles, blocks, 148)
            assert blocks % s == 0 and (s == 1 or tiles * s <= 148)


@pytest.mark.parametrize("t", ["Q4_K", "Q5_K", "Q6_K"])
def test_deep_products_of_64_rows_turn_every_ring_over(t):
    """Fourteen super-blocks through raw rings of four to six slots, an odd one with Q5_K, of which each group of expanders waits
    for every second slot; a slot that was read a turn early would bring another super-block's weights."""
    from bloomery_b200.ops import gemm as G
    N, K, rows = 200, 14 * 256, 64
    qw, ref_w = _weight(t, (N,), K, 5)
    torch.manual_seed(6)
    X = (torch.randn(rows, K, device=DEV) * 0.5).bfloat16()
    st, tiles = _status(), G.TileTable.dense(rows, DEV, 64)
    C = torch.full((40, rows, N), float("nan"), device=DEV)
    for c in C:
        G.qgemm(X, qw, tiles, out_f32=c, status=st)
    torch.cuda.synchronize()
    assert int(st) == 0
    # scales and offsets rounded to bf16: 2^-9 of terms of about 0.1 on each of K weights, times 0.5, added up at random
    assert torch.allclose(C[0], X.float() @ ref_w.bfloat16().float().T, rtol=1e-2, atol=6e-2)
    assert [i for i, c in enumerate(C) if not torch.equal(c, C[0])] == []
