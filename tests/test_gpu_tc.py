"""tcgen05 tensor-core path (16-bit B): parity with the oracle.

Bit tiles are expanded to exact 0/1 BF16/FP16 operands and products by 1 are
exact, so integer-valued B must give identical results; for N(0,1) B the
FP32 accumulation order differs from the oracle's, and every element is
checked against FP64 relative to its summation scale (≤ 1e-4), well inside
the 1e-2 bound of the precision form."""
import os

import numpy as np
import pytest
import torch

import oracle as O
from bitwise_spgemm_gb300 import capi, ops
from bitwise_spgemm_gb300 import workloads as W
from gpu_util import bf16_dev, words_dev

pytestmark = pytest.mark.gpu
TOL = 1e-4


@pytest.fixture
def force_tc():
    old = os.environ.get("BSP_TC")
    os.environ["BSP_TC"] = "1"
    yield
    if old is None:
        del os.environ["BSP_TC"]
    else:
        os.environ["BSP_TC"] = old


def _b16(Bf, kind):
    if kind == "bf16":
        b = W.f32_to_bf16_bits(Bf)
        return bf16_dev(b), W.bf16_bits_to_f32(b)
    t = torch.from_numpy(Bf).half().cuda()
    return t, t.float().cpu().numpy()


@pytest.mark.parametrize("kind", ["bf16", "f16"])
@pytest.mark.parametrize("M,K,N,p", [(128, 32, 256, 0.3), (300, 200, 264, 0.2), (1000, 1000, 512, 0.05),
                                     (77, 64, 8, 0.5), (512, 2048, 1024, 0.01)])
def test_tc_random(force_tc, kind, M, K, N, p):
    rng = np.random.default_rng(M + K + N)
    bits = rng.random((M, K)) < p
    if K >= 128:
        bits[: min(M, 130), 64:128] = False  # K tiles 2-3 empty for the first row block
    words = W.pack_bits(bits)
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    Bf = rng.standard_normal((K, N)).astype(np.float32)
    B, Bexact = _b16(Bf, kind)
    C = ops.spmm(wd, K, B, plan=plan).cpu().numpy()
    assert capi.device_status() == 0
    mx, mean, _ = O.rel_errors(C, O.spmm_f64(words, K, Bexact), O.spmm_abs_f64(words, K, Bexact))
    assert mx <= TOL, (mx, mean)
    # integer-valued B: exact
    Bi = rng.integers(-8, 9, (K, N)).astype(np.float32)
    Bt, Bie = _b16(Bi, kind)
    Ci = ops.spmm(wd, K, Bt, plan=plan).cpu().numpy()
    assert np.array_equal(Ci.astype(np.float64), O.spmm_f64(words, K, Bie))


def test_tc_block_structured_sample():
    """Block-structured A (32x32 tiles present w.p. 0.3, bits 0.8), the
    tensor-core workload at a reduced size, through the default dispatch."""
    A, present = W.block_bits(2048, 4096, p_tile=0.3, p_bit=0.8, seed=5)
    words = W.pack_bits(A)
    wd = words_dev(words)
    plan = ops.Plan(wd, 4096)
    rng = np.random.default_rng(6)
    Bf = rng.standard_normal((4096, 768)).astype(np.float32)
    B, Bexact = _b16(Bf, "bf16")
    C = ops.spmm(wd, 4096, B, plan=plan).cpu().numpy()
    assert capi.device_status() == 0
    mx, _, _ = O.rel_errors(C, O.spmm_f64(words, 4096, Bexact), O.spmm_abs_f64(words, 4096, Bexact))
    assert mx <= TOL
    # the CUDA-core walk agrees
    os.environ["BSP_TC"] = "0"
    try:
        C2 = ops.spmm(wd, 4096, B, plan=plan).cpu().numpy()
    finally:
        del os.environ["BSP_TC"]
    assert np.abs(C - C2).max() <= 1e-4 * max(1.0, np.abs(C2).max())


@pytest.mark.slow
def test_config3_full_size_row_sample():
    cfg = W.config3()
    words, K, N = cfg["words"], cfg["K"], cfg["N"]
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    B = bf16_dev(cfg["B"])
    C = ops.spmm(wd, K, B, plan=plan)
    assert capi.device_status() == 0
    Bexact = W.bf16_bits_to_f32(cfg["B"])
    rows = np.r_[0:128, 8192:8256, 16320:16384]
    Cs = C[torch.from_numpy(rows).cuda()].cpu().numpy()
    C64 = O.spmm_f64(words[rows], K, Bexact)
    mx, _, mxn = O.rel_errors(Cs, C64, O.spmm_abs_f64(words[rows], K, Bexact))
    assert mx <= TOL and mxn <= 1e-2


@pytest.mark.parametrize("M,K,N,p", [(512, 8192, 256, 0.3), (300, 4096, 40, 0.1), (256, 16384, 512, 0.02)])
def test_tc_split_k(force_tc, M, K, N, p):
    # few output tiles and a long reduction: with the preferred workspace the
    # occupied K tiles are split over several CTAs and the partials added in
    # a fixed order; the minimum workspace keeps one CTA per output tile
    rng = np.random.default_rng(M + K)
    words = W.pack_bits(rng.random((M, K)) < p)
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    assert plan.workspace_bytes(N) > plan.workspace_bytes(N, preferred=False)
    Bi = rng.integers(-8, 9, (K, N)).astype(np.float32)
    Bt, Bie = _b16(Bi, "bf16")
    ref = O.spmm_f64(words, K, Bie)
    C1 = ops.spmm(wd, K, Bt, plan=plan).cpu().numpy()  # split
    ws0 = torch.empty(max(plan.workspace_bytes(N, preferred=False), 1), dtype=torch.uint8, device="cuda")
    C0 = ops.spmm(wd, K, Bt, plan=plan, workspace=ws0).cpu().numpy()  # no split
    assert capi.device_status() == 0
    assert np.array_equal(C1.astype(np.float64), ref) and np.array_equal(C0.astype(np.float64), ref)
    # N(0,1) B: both orders within the precision-form tolerance, split run to run identical
    Bf = rng.standard_normal((K, N)).astype(np.float32)
    B, Bexact = _b16(Bf, "bf16")
    Ca = ops.spmm(wd, K, B, plan=plan).cpu().numpy()
    Cb = ops.spmm(wd, K, B, plan=plan).cpu().numpy()
    assert np.array_equal(Ca, Cb)
    mx, _, _ = O.rel_errors(Ca, O.spmm_f64(words, K, Bexact), O.spmm_abs_f64(words, K, Bexact))
    assert mx <= TOL, mx


@pytest.mark.parametrize("M,K,N", [(300, 200, 264), (1000, 1000, 512), (513, 4096, 776), (64, 40, 8),
                                   (8200, 300, 72), (600, 8300, 40)])
def test_tiled_b_matches_tensor_boxes(force_tc, M, K, N):
    # the preferred workspace copies B (and G) into tile order, one bulk copy
    # per tile, where the output has many row blocks; the minimum keeps TMA
    # tensor boxes.  The shared-memory bytes are the same, so integer-valued
    # operands (exact in any order) give identical results, including ragged
    # edges (K and M tails, a last column block of 8 or 8 < n < 64 columns);
    # N(0,1) operands stay within the precision-form tolerance either way.
    rng = np.random.default_rng(M + 3 * K + N)
    bits = rng.random((M, K)) < 0.2
    words = W.pack_bits(bits)
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    ws_pref = torch.empty(plan.workspace_bytes(N), dtype=torch.uint8, device="cuda")
    ws_min = torch.empty(max(plan.workspace_bytes(N, preferred=False), 1), dtype=torch.uint8, device="cuda")
    Bi, Bie = _b16(rng.integers(-8, 9, (K, N)).astype(np.float32), "bf16")
    ref = O.spmm_f64(words, K, Bie)
    for ws in (ws_pref, ws_min):
        assert np.array_equal(ops.spmm(wd, K, Bi, plan=plan, workspace=ws).cpu().numpy().astype(np.float64), ref)
    B, Bexact = _b16(rng.standard_normal((K, N)).astype(np.float32), "bf16")
    for ws in (ws_pref, ws_min):
        C = ops.spmm(wd, K, B, plan=plan, workspace=ws).cpu().numpy()
        mx, _, _ = O.rel_errors(C, O.spmm_f64(words, K, Bexact), O.spmm_abs_f64(words, K, Bexact))
        assert mx <= TOL
    assert capi.device_status() == 0
    # transposed product: G [M][N] tiled over M
    n_min, n_pref = _t_workspaces(M, K, N)
    Gi, Gie = _b16(rng.integers(-8, 9, (M, N)).astype(np.float32), "bf16")
    ref_t = O.spmm_t_f64(words, M, K, Gie)
    for nb in (n_pref, n_min):
        ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
        dX = ops.spmm_t(wd, M, K, Gi, plan=plan, workspace=ws).cpu().numpy()
        assert np.array_equal(dX.astype(np.float64), ref_t)
    assert capi.device_status() == 0


def _t_workspaces(M, K, N):
    import ctypes
    a, b = ctypes.c_size_t(), ctypes.c_size_t()
    capi.call("bsp_spmm_t_workspace", M, K, ctypes.byref(a))
    capi.call("bsp_spmm_t_workspace_preferred", M, K, N, ctypes.byref(b))
    assert b.value >= a.value
    return a.value, b.value


@pytest.mark.parametrize("kind", ["bf16", "f16"])
@pytest.mark.parametrize("M,K,N", [(1, 32, 8), (127, 31, 64), (128, 33, 72), (129, 96, 128), (256, 128, 136),
                                   (257, 160, 192), (385, 300, 264), (5000, 200, 1500), (200, 5000, 1500)])
def test_tc_items_and_stages(force_tc, kind, M, K, N):
    """Edges of the 256x128 items and of the stages of four K tiles, empty
    tiles and halves, one item and many per CTA: exact on integers, both ways."""
    rng = np.random.default_rng(M + K + N)
    bits = rng.random((M, K)) < 0.2
    bits[128:256] = False          # a half without bits
    bits[:, 32:64] = False         # a K tile without bits
    bits[: M // 2, K // 2:] = False
    words = W.pack_bits(bits)
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    Bi, Bie = _b16(rng.integers(-8, 9, (K, N)).astype(np.float32), kind)
    C = ops.spmm(wd, K, Bi, plan=plan).cpu().numpy()
    assert np.array_equal(C.astype(np.float64), O.spmm_f64(words, K, Bie))
    Gi, Gie = _b16(rng.integers(-8, 9, (M, N)).astype(np.float32), kind)
    dX = ops.spmm_t(wd, M, K, Gi, plan=plan).cpu().numpy()
    assert np.array_equal(dX.astype(np.float64), O.spmm_t_f64(words, M, K, Gie))
    assert capi.device_status() == 0


@pytest.mark.parametrize("kind", ["bf16", "f16"])
@pytest.mark.parametrize("M,K,N", [(300, 200, 1), (700, 3000, 133), (600, 4000, 500), (128, 8192, 129)])
def test_tc_unaligned_columns(force_tc, kind, M, K, N):
    """Widths without 16-byte rows go through tile order (with and without
    split-K); nothing is written past N, and a value that is not finite
    reaches only the rows that hold its column."""
    rng = np.random.default_rng(M + K + N)
    bits = rng.random((M, K)) < 0.3
    words = W.pack_bits(bits)
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    Bi, Bie = _b16(rng.integers(-8, 9, (K, N)).astype(np.float32), kind)
    ref = O.spmm_f64(words, K, Bie)
    out = torch.full((M, N + 3), 7.0, device="cuda")
    ops.spmm(wd, K, Bi, plan=plan, out=out[:, :N])
    assert np.array_equal(out[:, :N].cpu().numpy().astype(np.float64), ref)
    assert torch.all(out[:, N:] == 7.0)
    for bad in (float("inf"), float("nan")):
        B = Bi.clone()
        B[5, N // 2] = bad
        C = ops.spmm(wd, K, B, plan=plan).cpu().numpy()
        hit = np.zeros((M, N), dtype=bool)
        hit[bits[:, 5], N // 2] = True
        assert np.array_equal(~np.isfinite(C), hit)
        assert np.array_equal(C[~hit].astype(np.float64), ref[~hit])
    assert capi.device_status() == 0


@pytest.mark.parametrize("kind", ["bf16", "f16"])
@pytest.mark.parametrize("M,K,N,p", [(8200, 1000, 264, 0.05), (8448, 3000, 64, 0.01)])
def test_three_tile_stages(force_tc, kind, M, K, N, p):
    # 32+ row blocks: stages of three K tiles (two stages in flight); list
    # lengths that are not multiples of three leave a short last stage
    rng = np.random.default_rng(M + K)
    bits = rng.random((M, K)) < p
    bits[:300, 96:320] = False  # a run of empty K tiles for the first row blocks
    words = W.pack_bits(bits)
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    Bi, Bie = _b16(rng.integers(-8, 9, (K, N)).astype(np.float32), kind)
    C = ops.spmm(wd, K, Bi, plan=plan).cpu().numpy()
    assert capi.device_status() == 0
    assert np.array_equal(C.astype(np.float64), O.spmm_f64(words, K, Bie))
    B, Bexact = _b16(rng.standard_normal((K, N)).astype(np.float32), kind)
    C = ops.spmm(wd, K, B, plan=plan).cpu().numpy()
    mx, _, _ = O.rel_errors(C, O.spmm_f64(words, K, Bexact), O.spmm_abs_f64(words, K, Bexact))
    assert mx <= TOL


@pytest.mark.parametrize("M,K,N,p", [(1, 33, 1, 0.5), (128, 64, 8, 0.3), (257, 129, 43, 0.2), (300, 1000, 201, 0.2),
                                     (64, 4096, 256, 0.3), (4096, 64, 40, 0.3), (1000, 3000, 520, 0.1)])
def test_f32_parts(force_tc, M, K, N, p):
    """FP32 operands as three BF16 parts: exact where the sums are (integers of
    13 bits, |sum| < 2^24), otherwise within the bound of truncating sums of 16
    products each; a value outside the parts' range, or values of very different
    sizes, leave the whole product to the walk."""
    rng = np.random.default_rng(M + K + N)
    bits = rng.random((M, K)) < p
    words = W.pack_bits(bits)
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    pad = 3 if N % 2 else 0
    mk = lambda a: torch.nn.functional.pad(torch.from_numpy(a), (0, pad)).cuda()[:, :N]
    B, G = rng.integers(-4000, 4001, (K, N)).astype(np.float32), rng.integers(-4000, 4001, (M, N)).astype(np.float32)
    out = torch.full((M, N + 5), 7.0, device="cuda")
    ops.spmm(wd, K, mk(B), plan=plan, out=out[:, :N])
    assert np.array_equal(out[:, :N].cpu().numpy().astype(np.float64), O.spmm_f64(words, K, B))
    assert torch.all(out[:, N:] == 7.0)
    dX = ops.spmm_t(wd, M, K, mk(G), plan=plan).cpu().numpy()
    assert np.array_equal(dX.astype(np.float64), O.spmm_t_f64(words, M, K, G))
    B, G = rng.standard_normal((K, N)).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32)
    C = ops.spmm(wd, K, mk(B), plan=plan).cpu().numpy()
    err = np.abs(C - O.spmm_f64(words, K, B))
    # each of ceil(K/16) steps loses at most 2 units of 2^-23 of the sum so far
    assert np.all(err <= (-(-K // 16) + 4) * 2.0**-22 * O.spmm_abs_f64(words, K, B) + 1e-30)
    dX = ops.spmm_t(wd, M, K, mk(G), plan=plan).cpu().numpy()
    assert np.all(np.abs(dX - O.spmm_t_f64(words, M, K, G))
                  <= (-(-M // 16) + 4) * 2.0**-22 * (bits.T.astype(np.float64) @ np.abs(G)) + 1e-30)
    heavy = np.exp(6 * rng.standard_normal(max(M, K) * N)).astype(np.float32)  # sums that lose bits by truncation
    for bad in (float("inf"), float("nan"), 1e38, 1e-38, None):
        if bad is None:
            if min(M, K) * N < 1000:
                continue
            B, G = heavy[:K * N].reshape(K, N), heavy[:M * N].reshape(M, N)
        else:
            B[K // 2, N // 2] = bad
            G[M // 2, N // 2] = bad
        got = ops.spmm(wd, K, mk(B), plan=plan), ops.spmm_t(wd, M, K, mk(G), plan=plan)
        os.environ["BSP_TC"] = "0"
        want = ops.spmm(wd, K, mk(B), plan=plan), ops.spmm_t(wd, M, K, mk(G), plan=plan)
        os.environ["BSP_TC"] = "1"
        for g, w in zip(got, want):
            assert torch.equal(g.view(torch.int32), w.view(torch.int32))
    assert capi.device_status() == 0


@pytest.mark.parametrize("kind", ["bf16", "f16"])
@pytest.mark.parametrize("M,K,N,direct", [(300, 2600, 1000, True), (129, 10000, 264, True), (64, 20000, 8, True),
                                          (700, 500, 200, True), (2000, 500, 200, False),
                                          (300, 2600, 1001, False)])
def test_spmm_t_in_16_bits(force_tc, kind, M, K, N, direct):
    """dX in G's type: the FP32 result rounded once, whether the epilogue rounds
    it or (split reductions, unaligned rows) a cast afterwards; row and column
    remainders of the boxes, blocks of dX without a bit."""
    rng = np.random.default_rng(M + K + N)
    bits = rng.random((M, K)) < 0.1
    bits[:, 256:640] = False
    wd = words_dev(W.pack_bits(bits))
    plan = ops.Plan(wd, K)
    G, _ = _b16(rng.standard_normal((M, N)).astype(np.float32), kind)
    want = ops.spmm_t(wd, M, K, G, plan=plan).to(G.dtype)
    got = ops._spmm_t_as(wd, M, K, G, plan, None, G.dtype)
    assert (got is not None) == direct
    if direct:
        assert torch.equal(got, want)
    assert torch.equal(ops.spmm_t(wd, M, K, G, plan=plan, dtype=G.dtype), want)
    assert capi.device_status() == 0


def test_widths_past_65535_column_blocks(force_tc):
    """More blocks of 128 columns than a grid's y holds: the product, Aᵀ·G and,
    for rows without 16-byte access, the prototype plan and the walk."""
    N = 65535 * 128 + 136
    rng = np.random.default_rng(3)
    bits = rng.random((3, 40)) < 0.4
    bits[:, 7] = True
    wd = words_dev(W.pack_bits(bits))
    plan = ops.Plan(wd, 40)
    g = torch.Generator(device="cuda").manual_seed(5)
    A = torch.from_numpy(bits.astype(np.float32)).cuda()
    B = torch.randint(-8, 9, (40, N), device="cuda", generator=g).bfloat16()
    assert torch.equal(ops.spmm(wd, 40, B, plan=plan), A @ B.float())
    dX = ops.spmm_t(wd, 3, 40, B[:3], plan=plan)
    assert torch.equal(dX, A.T @ B[:3].float())
    del B, dX
    rows = np.repeat(rng.random((1, 64)) < 0.5, 8, 0)
    rows[3, 11] ^= True
    wd = words_dev(W.pack_bits(rows))
    plan = ops.Plan(wd, 64, mode=capi.PLAN_PROTO)
    assert plan.info()["mode"] == capi.PLAN_PROTO
    A = torch.from_numpy(rows.astype(np.float32)).cuda()
    Bf = torch.randint(-8, 9, (64, N + 1), device="cuda", generator=g).float()
    out = torch.full((8, N + 1), 7.0, device="cuda")
    os.environ["BSP_TC"] = "0"
    ops.spmm(wd, 64, Bf, plan=plan, out=out)
    os.environ["BSP_TC"] = "1"
    assert torch.equal(out, A @ Bf)
    assert capi.device_status() == 0


@pytest.mark.parametrize("kind", ["bf16", "f16"])
@pytest.mark.parametrize("M,K,N", [(130, 512, 132), (300, 2600, 264), (2100, 1700, 1296), (257, 8192, 8)])
def test_tc_segments(force_tc, kind, M, K, N):
    """Column slices of a wider B (tile order, sums handed over every 16 K
    tiles): segments without tiles, halves with tiles in some segments only,
    with and without split-K, C by TMA and by plain stores; exact on integers."""
    rng = np.random.default_rng(M + K + N)
    bits = rng.random((M, K)) < 0.2
    bits[:128, 256:1100] = False
    bits[128:, 600:900] = False
    bits[256:, :300] = False
    words = W.pack_bits(bits)
    wd = words_dev(words)
    plan = ops.Plan(wd, K)
    wide, exact = _b16(rng.integers(-8, 9, (K, N + 5)).astype(np.float32), kind)
    ref = O.spmm_f64(words, K, np.ascontiguousarray(exact[:, 3:N + 3]))
    ws = torch.empty(plan.workspace_bytes(N + 1) + (1 << 24), dtype=torch.uint8, device="cuda")
    for pad in (0, 4, 3):
        out = torch.full((M, N + pad), 7.0, device="cuda")
        ops.spmm(wd, K, wide[:, 3:N + 3], plan=plan, out=out[:, :N], workspace=ws)
        assert np.array_equal(out[:, :N].cpu().numpy().astype(np.float64), ref)
        assert torch.all(out[:, N:] == 7.0)
    assert capi.device_status() == 0


def test_tc_unaligned_columns_of_tiny_values(force_tc):
    """BF16 values below 2^-100, whose sums may be subnormal: the walk's bits."""
    rng = np.random.default_rng(4)
    M, K, N = 300, 1500, 67
    wd = words_dev(W.pack_bits(rng.random((M, K)) < 0.2))
    B = torch.from_numpy((rng.standard_normal((K, N)) * 2.0 ** -128).astype(np.float32)).cuda().bfloat16()
    C = ops.spmm(wd, K, B, plan=ops.Plan(wd, K))
    assert torch.equal(C.view(torch.int32), ops.spmm(wd, K, B).view(torch.int32)) and bool((C != 0).any())


def _frobenius(C, want):
    return float((C.double() - want).norm() / want.norm())


@pytest.mark.parametrize("kind", ["bf16", "f16"])
@pytest.mark.parametrize("M,K,N,p", [(2048, 8192, 1281, 0.24), (3000, 4096, 901, 0.1), (8200, 2048, 301, 0.2)])
def test_tc_unaligned_columns_lose_no_precision(force_tc, kind, M, K, N, p):
    """Widths without 16-byte rows: N(0,1) products no further from FP64 than
    the walk's sums (the outputs are wide enough to run without split-K)."""
    g = torch.Generator(device="cuda").manual_seed(M)
    A = torch.rand((M, K), device="cuda", generator=g) < p
    wd = ops.pack_rows(A.to(torch.uint8))
    plan = ops.Plan(wd, K)
    B = torch.randn((K, N), device="cuda", generator=g).to(torch.bfloat16 if kind == "bf16" else torch.float16)
    want = A.double() @ B.double()
    C = ops.spmm(wd, K, B, plan=plan)
    os.environ["BSP_TC"] = "0"
    walk = ops.spmm(wd, K, B, plan=plan)
    os.environ["BSP_TC"] = "1"
    assert not torch.equal(C, walk)  # the tensor cores did run
    assert _frobenius(C, want) <= _frobenius(walk, want)


def test_tc_unaligned_columns_with_compensated_rows(force_tc):
    """A row of more than 4096 set bits: the walk's compensated sums."""
    g = torch.Generator(device="cuda").manual_seed(8)
    M, K, N = 300, 12000, 129
    A = torch.rand((M, K), device="cuda", generator=g) < 0.3
    A[17] = torch.rand(K, device="cuda", generator=g) < 0.6
    wd = ops.pack_rows(A.to(torch.uint8))
    B = torch.randn((K, N), device="cuda", generator=g).half()
    C = ops.spmm(wd, K, B, plan=ops.Plan(wd, K))
    assert torch.equal(C, ops.spmm(wd, K, B))
    # rounded once, and a compensated sum's 2^-24 of the error terms
    want = A[17].double() @ B.double()
    assert float((C[17].double() - want).abs().max()) <= 2.0 ** -23 * float(want.abs().max())


def _columns(kind, K, N, g):
    """FP32 values [K, N] of a kind, and whether the tensor cores' sums are exact enough for them."""
    rnd = lambda: torch.rand((K, N), device="cuda", generator=g)
    z = torch.randn((K, N), device="cuda", generator=g)
    two = lambda f, d: torch.where(rnd() < f, 2.0 ** -d, 1.0) * (1 + rnd())
    if kind == "normal":
        return z, True
    if kind == "lognormal":
        return torch.exp(z), True
    if kind == "outliers":
        z[K // 3, ::7] = 100.0
        return z, True
    if kind == "half 2^-11":
        return two(0.5, 11), None
    if kind == "two per cent 2^-14":
        return two(0.02, 14), None
    if kind == "half 2^-16":
        return two(0.5, 16), False
    if kind == "softmax gradient":
        p = torch.softmax(2 * z, 0)
        p[0] -= 1
        return p, False
    z[:, N // 2] = two(0.3, 16)[:, 0] * 2.0 ** -10  # one column of unequal values below the others
    return z, False


@pytest.mark.parametrize("kind", ["normal", "lognormal", "outliers", "half 2^-11", "two per cent 2^-14", "half 2^-16",
                                  "softmax gradient", "one column"])
@pytest.mark.parametrize("M,K,N,p", [(600, 512, 256, 0.1), (1500, 4096, 256, 0.1), (512, 4096, 1800, 0.95)])
def test_f32_parts_lose_no_precision(force_tc, kind, M, K, N, p):
    """FP32 products on the tensor cores: no further from FP64 than the walk's
    (its rounding is random, so by 3 %), whatever the values; the walk's bits where
    a column's values are too unequal."""
    g = torch.Generator(device="cuda").manual_seed(M)
    A = torch.rand((M, K), device="cuda", generator=g) < p
    wd = ops.pack_rows(A.to(torch.uint8))
    plan = ops.Plan(wd, K, mode=capi.PLAN_DIRECT)
    B, exact = _columns(kind, K, N, g)
    G, exact_t = _columns(kind, M, N, g)
    Ad = A.double()
    got = ops.spmm(wd, K, B, plan=plan), ops.spmm_t(wd, M, K, G, plan=plan)
    os.environ["BSP_TC"] = "0"
    walk = ops.spmm(wd, K, B, plan=plan), ops.spmm_t(wd, M, K, G, plan=plan)
    os.environ["BSP_TC"] = "1"
    for c, w, want, ex in zip(got, walk, (Ad @ B.double(), Ad.T @ G.double()), (exact, exact_t)):
        assert _frobenius(c, want) <= 1.03 * _frobenius(w, want)
        if ex is not None:
            assert torch.equal(c, w) == (not ex)
    assert capi.device_status() == 0


@pytest.mark.parametrize("M,K,N", [(300, 4096, 64), (64, 500, 257), (3000, 96, 40)])
def test_f32_parts_of_long_integers(force_tc, M, K, N):
    """Integers of 22 bits, which take all three parts, at most three a sum: exact."""
    rng = np.random.default_rng(M + K)
    bits = np.zeros((M, K), dtype=bool)
    for i in range(M):
        bits[i, rng.choice(K, 3, replace=False)] = True
    words = W.pack_bits(bits)
    wd = words_dev(words)
    B = rng.integers(-(1 << 22), 1 << 22, (K, N)).astype(np.float32)
    C = ops.spmm(wd, K, torch.from_numpy(B).cuda(), plan=ops.Plan(wd, K, mode=capi.PLAN_DIRECT))
    assert np.array_equal(C.cpu().numpy().astype(np.float64), O.spmm_f64(words, K, B))
    cols = W.pack_bits(np.ascontiguousarray(bits.T))
    G = rng.integers(-(1 << 22), 1 << 22, (K, N)).astype(np.float32)
    wt = words_dev(cols)
    dX = ops.spmm_t(wt, K, M, torch.from_numpy(G).cuda(), plan=ops.Plan(wt, M, mode=capi.PLAN_DIRECT))
    assert np.array_equal(dX.cpu().numpy().astype(np.float64), O.spmm_f64(words, K, G))
    assert capi.device_status() == 0


def test_workspace_of_column_slices():
    """Rows of B off the 16-byte grid, N a multiple of 8: the workspace that is
    asked for lets a dense product use the tensor cores, and is empty for a small
    one, which uses none."""
    import ctypes
    g = torch.Generator(device="cuda").manual_seed(2)

    def layout(plan, K, N, B):
        n = ctypes.c_size_t()
        capi.call("bsp_spmm_workspace_layout", plan.handle, K, N, B.data_ptr(),
                  capi.F32 if B.dtype == torch.float32 else capi.BF16, B.stride(0), ctypes.byref(n))
        return n.value

    for M, K, N in [(600, 2048, 512), (2600, 2048, 1024)]:  # with a split reduction, and without
        A = torch.rand((M, K), device="cuda", generator=g) < 0.3
        wd = ops.pack_rows(A.to(torch.uint8))
        plan = ops.Plan(wd, K, mode=capi.PLAN_DIRECT)
        B = torch.randn((K, N + 5), device="cuda", generator=g).bfloat16()[:, 3:N + 3]
        C = ops.spmm(wd, K, B, plan=plan)
        assert not torch.equal(C, ops.spmm(wd, K, B))  # not the walk's sums
        assert float((C - A.float() @ B.float()).abs().max()) <= 1e-3
    A = torch.rand((64, 96), device="cuda", generator=g) < 0.1
    wd = ops.pack_rows(A.to(torch.uint8))
    plan = ops.Plan(wd, 96, mode=capi.PLAN_DIRECT)
    for B in (torch.randn((96, 21), device="cuda").bfloat16()[:, 3:19], torch.randn((96, 17), device="cuda")):
        assert layout(plan, 96, B.shape[1], B) == 0
        assert torch.equal(ops.spmm(wd, 96, B, plan=plan), ops.spmm(wd, 96, B))


def test_spmm_t_in_16_bits_asks_before_it_allocates(force_tc, monkeypatch):
    """Where the library has no 16-bit pass (a split reduction, rows off the
    grid) nothing is allocated for it."""
    g = torch.Generator(device="cuda").manual_seed(3)
    cases = []
    for M, K, N in [(2000, 500, 200), (300, 2600, 1001)]:
        wd = ops.pack_rows((torch.rand((M, K), device="cuda", generator=g) < 0.1).to(torch.uint8))
        cases.append((wd, M, K, torch.randn((M, N), device="cuda", generator=g).bfloat16(), ops.Plan(wd, K)))

    def refuse(*a, **k):
        raise AssertionError("allocated")

    monkeypatch.setattr(torch, "empty", refuse)
    for wd, M, K, G, plan in cases:
        assert ops._spmm_t_as(wd, M, K, G, plan, None, G.dtype) is None


def test_products_on_a_nearly_full_gpu(monkeypatch):
    """Where the preferred workspace cannot be had, the products run in the
    minimum: as they did before they knew of parts, copies and splits."""
    g = torch.Generator(device="cuda").manual_seed(4)
    M, K, N = 1024, 2048, 512
    A = torch.rand((M, K), device="cuda", generator=g) < 0.2
    wd = ops.pack_rows(A.to(torch.uint8))
    plan = ops.Plan(wd, K, mode=capi.PLAN_DIRECT)
    real = torch.empty

    def empty(*size, **kw):
        if kw.get("dtype") == torch.uint8 and size[0] > 1 << 20:
            raise torch.OutOfMemoryError("full")
        return real(*size, **kw)

    for dt, width in ((torch.float32, N), (torch.bfloat16, N), (torch.bfloat16, N + 1)):
        B = torch.randint(-8, 9, (K, width), device="cuda", generator=g).to(dt)
        G = torch.randint(-8, 9, (M, width), device="cuda", generator=g).to(dt)
        with monkeypatch.context() as m:
            m.setattr(torch, "empty", empty)
            C, dX = ops.spmm(wd, K, B, plan=plan), ops.spmm_t(wd, M, K, G, plan=plan)
            dX16 = ops.spmm_t(wd, M, K, G, plan=plan, dtype=dt)
        assert torch.equal(C, A.float() @ B.float()) and torch.equal(dX, A.float().T @ G.float())
        assert torch.equal(dX16, dX.to(dt))
    W8 = torch.randint(-8, 9, (M, K), device="cuda", generator=g).to(torch.int8)
    mat = ops.Int8Matrix(W8)
    B = torch.randint(-8, 9, (K, N), device="cuda", generator=g).bfloat16()
    with monkeypatch.context() as m:
        m.setattr(torch, "empty", empty)
        C = mat.matmul(B)
    assert torch.equal(C, W8.float() @ B.float())
    assert capi.device_status() == 0
