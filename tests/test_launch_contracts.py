"""Launch contracts of the CUDA library, exercised without a card: every entry point checks shapes, types, alignment and
limits before it touches the device and answers a negative code (``BL_ERR_SHAPE`` -2, ``BL_ERR_TYPE`` -3,
``BL_ERR_ALIGN`` -4, ``BL_ERR_LIMIT`` -5) that ``bl_error_string`` names.  The pointers below are never dereferenced:
each call is refused first.  (The reference keeps the same kind of suite for its device contract,
``crates/device/src/fault.rs`` and the launch checks of ``crates/chain``.)"""
import ctypes

import pytest

from bloomery_b200.ops._lib import KernelError, check, cuda

SHAPE, TYPE, ALIGN, LIMIT = -2, -3, -4, -5
I, L, F, P = ctypes.c_int, ctypes.c_long, ctypes.c_float, ctypes.c_void_p
A = 0x10000          # an aligned address nothing reads
WT_Q4_K, WT_F32, WT_FP8_B128 = 12, 0, 41


def _qgemm(K=1024, N=256, wtype=WT_Q4_K, tile_rows=32, x=A, ldx=None, c_f32=A, c_bf16=0, rows=64):
    return cuda().bl_qgemm(P(x), L(K if ldx is None else ldx), L(rows), P(A), P(0), I(wtype), I(1), I(N), I(K), P(A), P(A), I(4),
                           I(tile_rows), P(c_f32), P(c_bf16), L(N), P(0), P(0), P(0), L(0), P(0), I(148), P(0))


def test_quantised_gemm_refuses_before_it_launches():
    assert _qgemm(K=1000) == SHAPE                    # K not a multiple of 256
    assert _qgemm(tile_rows=48) == SHAPE
    assert _qgemm(c_f32=A, c_bf16=A) == SHAPE         # exactly one output
    assert _qgemm(c_f32=0, c_bf16=0) == SHAPE
    assert _qgemm(x=A + 2) == ALIGN
    assert _qgemm(ldx=1028) == ALIGN                  # rows of X not 16-byte multiples
    assert _qgemm(wtype=WT_F32) == TYPE               # float rows have no expander
    assert _qgemm(wtype=99) == TYPE
    assert cuda().bl_qgemm_supports(I(WT_Q4_K)) == 1 and cuda().bl_qgemm_supports(I(WT_FP8_B128)) == 1
    assert cuda().bl_qgemm_supports(I(WT_F32)) == 0


def test_forms_of_a_weight_that_the_quantised_gemm_has_no_kernel_for_are_refused():
    def call(form, tile_rows, pair):
        return cuda().bl_qgemm_split(P(A), L(1024), L(64), P(A), P(A if pair else 0), I(WT_Q4_K), I(1), I(256), I(1024), P(A), P(A), I(4),
                                     I(tile_rows), P(A), P(0), L(256), P(0), P(0), P(0), L(0), P(0), I(148), I(0), I(form), I(1),
                                     P(0), P(0), P(0))
    assert call(3, 32, False) == SHAPE and call(-1, 32, False) == SHAPE
    assert call(2, 128, False) == SHAPE and call(2, 64, True) == SHAPE and call(2, 128, True) == SHAPE


def _fp8_gemm(K=1024, tile_rows=32, x=A, ldx=None, c_f32=A, c_bf16=0):
    return cuda().bl_fp8_gemm(P(x), L(K if ldx is None else ldx), L(64), P(A), P(A), P(0), I(1), I(256), I(K), P(A), P(A), I(4),
                              I(tile_rows), P(c_f32), P(c_bf16), L(256), P(0), P(0), P(0), L(0), P(0), I(148), P(0))


def test_block_scaled_fp8_entries_refuse_before_they_launch():
    assert _fp8_gemm(K=1000) == SHAPE
    assert _fp8_gemm(tile_rows=64) == SHAPE           # this kernel takes 32-token tiles only
    assert _fp8_gemm(c_f32=A, c_bf16=A) == SHAPE
    assert _fp8_gemm(x=A + 4) == ALIGN
    assert _fp8_gemm(ldx=1000) == ALIGN
    rows = lambda **kw: cuda().bl_fp8_rows(P(kw.get("x", A)), I(kw.get("f32", 0)), L(kw.get("ldx", 1024)), P(kw.get("gain", 0)), F(1e-6),  # noqa: E731
                                           I(kw.get("M", 4)), I(kw.get("K", 1024)), P(A), L(kw.get("ldc", 1024)), P(A), P(0))
    assert rows(K=1000) == SHAPE and rows(M=0) == SHAPE and rows(ldc=1000) == SHAPE
    assert rows(x=A + 8) == ALIGN
    assert rows(gain=A, f32=0) == TYPE                # the fused norm reads fp32 rows


def test_attention_and_router_entries_refuse_before_they_launch():
    lib = cuda()
    kv = lambda lora, rope, M: lib.bl_mla_kv_append(P(A), L(576), P(A), P(A), F(1e-6), I(lora), I(rope), I(M), P(A), P(A), P(A),  # noqa: E731
                                                    I(4), I(16), P(A), P(A), I(0), P(0))
    assert kv(256, 64, 1) == SHAPE and kv(512, 32, 1) == SHAPE and kv(512, 64, 0) == SHAPE
    router = lambda E, K, M, wt: lib.bl_router(P(A), L(K), P(A), F(1e-6), P(A), I(wt), I(K), I(E), I(M), P(A), P(0), P(0), P(0),  # noqa: E731
                                               P(0), P(A), I(0), P(0), P(0), I(8), I(0), I(1), F(1.0), I(1), I(1), P(0), P(0), P(0),
                                               P(0), P(0), P(0), L(0), L(0), P(0), P(0))
    assert router(100000, 2048, 1, WT_F32) == LIMIT   # more experts than the routing block holds
    assert router(128, 1000, 1, WT_F32) == SHAPE
    assert router(128, 2048, 1, WT_Q4_K) == TYPE      # router weights are float rows


def test_every_code_has_a_name_and_check_raises_it():
    names = {code: cuda().bl_error_string(I(code)).decode() for code in (SHAPE, TYPE, ALIGN, LIMIT)}
    assert len(set(names.values())) == 4 and all(names.values())
    with pytest.raises(KernelError, match=r"bl_qgemm: .* \(code -2\)"):
        check(_qgemm(K=1000), "bl_qgemm")
    check(0, "nothing")


def test_a_tile_table_that_a_launch_writes_is_no_longer_fixed(monkeypatch):
    """qgemm takes a fixed table's tile count from the host and reads the table before the launch in front of it ends."""
    import torch
    from types import SimpleNamespace
    from bloomery_b200.ops import gemm as G
    done = lambda *a: 0                                                                                  # noqa: E731
    monkeypatch.setattr(G, "cuda", lambda: SimpleNamespace(bl_gemm_build_tiles=done, bl_gemm_build_tiles_causal=done, bl_moe_plan=done))
    monkeypatch.setattr(G, "stream", lambda: P(0))
    rows = torch.tensor([70], dtype=torch.int32)
    for again in (lambda t: t.build(rows), lambda t: t.build(rows, causal_pos0=0, causal_kind=1),
                  lambda t: G.moe_plan(rows, rows.float(), 1, t, rows, rows, rows.float())):
        t = G.TileTable.dense(70, "cpu", 32)
        assert t.fixed == 3
        again(t)
        assert t.fixed == 0


def _gemv_plan(M, K, reduce=0, norm=1, rows=(4096, 512, 512), types=(12, 12, 14)):
    """Blocks, weight rows and units a lane takes at a time, rows as a whole, bytes of shared memory on 148 processors."""
    out = (ctypes.c_long * 5)()
    n = len(rows)
    assert cuda().bl_gemv_plan(I(n), (I * n)(*rows), (I * n)(*types), I(K), I(M), I(norm), I(reduce), I(148), out) == 0
    return list(out)


def test_rows_behind_a_reduction_keep_several_weight_rows_in_flight():
    """A head of 151,936 rows gives a warp more of them than it takes at a time: three, or two beside eight rows' sums."""
    for M, R in ((1, 3), (2, 3), (3, 3), (4, 3), (5, 2), (8, 2)):
        assert _gemv_plan(M, 2048, reduce=1, rows=(151936,), types=(14,))[1:3] == [R, 1]
    assert _gemv_plan(8, 4096, reduce=1)[1:3] == [1, 2]                    # two columns of units a lane are needed there
    assert cuda().bl_gemv_plan(I(1), (I * 1)(64), (I * 1)(0), I(2048), I(1), I(0), I(0), I(148), (L * 5)()) == TYPE


def test_the_blocks_of_a_gemv_fit_a_processor_two_at_a_time():
    """They are counted as one wave of two a processor, whose blocks share 227 KB less 1 KB each: at any width of quantised rows, with
    or without the norm's fp32 rows, alone or behind a reduction."""
    for types in ((12, 12, 14), (40, 40, 40)):
        for K in range(256, 8193, 256):
            for M in range(1, 9):
                for kw in (dict(), dict(norm=0), dict(reduce=1)):
                    assert 2 * (_gemv_plan(M, K, types=types, **kw)[4] + 1024) <= 227 * 1024, (types, K, M, kw)


def test_rows_that_other_ranks_wait_for_are_not_left_out():
    from bloomery_b200.ops.decode import PushOut
    push = PushOut()
    push.n_ranks = 2
    assert cuda().bl_gemv(I(1), (P * 1)(A), (I * 1)(64), (I * 1)(WT_Q4_K), I(2048), I(4), I(0), P(0), L(0), P(0), F(1e-6), P(A), P(A),
                          P(A), L(64), P(0), L(0), P(0), ctypes.byref(push), P(0), I(0), I(148), I(0), P(0), P(0), P(A), P(0)) == SHAPE
