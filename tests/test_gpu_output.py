"""Output side and multi-bit operands on the GPU: symbolic output masks and
their first-fit grouping, bit-plane products and the int8 path, against the
oracle (source/src/transform.cuh:1028-1157 and :2199-2246, main.cu:895-910)."""
import numpy as np
import pytest
import torch

import oracle as O
from bitwise_spgemm_gb300 import capi, ops
from bitwise_spgemm_gb300 import workloads as W
from gpu_util import dev, words_dev, words_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N,pa,pb", [(300, 70, 90, 0.05, 0.1), (64, 4096, 5000, 0.002, 0.01),
                                         (1000, 33, 31, 0.2, 0.05), (5, 32, 8192, 0.5, 0.001),
                                         (128, 256, 1, 0.1, 0.5)])
def test_symbolic_rows_match_oracle(M, K, N, pa, pb):
    rng = np.random.default_rng(M * 7 + N)
    A = rng.random((M, K)) < pa
    A[M // 2] = False  # an empty row
    Bm = rng.random((K, N)) < pb
    a, b = W.pack_bits(A), W.pack_bits(Bm)
    got = words_host(ops.symbolic_rows(words_dev(a), K, words_dev(b), N))
    assert np.array_equal(got, O.symbolic_rows(a, K, b, N))
    # the mask is the nonzero pattern of the integer product
    prod = (A.astype(np.int64) @ Bm.astype(np.int64)) > 0
    assert np.array_equal(got, W.pack_bits(prod))


@pytest.mark.parametrize("N,pb", [(31, 0.05), (2056, 0.01), (8192, 0.002), (300, 0.3)])
def test_symbolic_rows_through_plan(N, pb):
    """Clustered A (plus rows that fit no cluster): the planned pass — the
    clusters' bit-sliced counts, then each row's added and removed columns —
    gives the same masks as the direct OR walk and the oracle, including
    dense B masks where counts run high and removed columns matter."""
    from bitwise_spgemm_gb300 import capi
    rng = np.random.default_rng(N)
    A, _, _ = W.clustered_bits(1500, 2500, n_proto=7, p_proto=0.08, p_flip=0.006, seed_proto=N, seed_rows=N + 1)
    A[::13] = rng.random((A[::13].shape[0], 2500)) < 0.03  # rows that fit no cluster
    A[5] = False                                             # an empty row
    Bm = rng.random((2500, N)) < pb
    a, b = W.pack_bits(A), W.pack_bits(Bm)
    ad, bd = words_dev(a), words_dev(b)
    plan = ops.Plan(ad, 2500, mode=capi.PLAN_PROTO)
    info = plan.info()
    assert info["mode"] == capi.PLAN_PROTO and info["direct_rows"] > 0 and info["delta_nnz"] > 0
    got = words_host(ops.symbolic_rows(ad, 2500, bd, N, plan=plan))
    assert np.array_equal(got, words_host(ops.symbolic_rows(ad, 2500, bd, N)))
    assert np.array_equal(got, O.symbolic_rows(a, 2500, b, N))
    assert capi.device_status() == 0


@pytest.mark.parametrize("TR,G", [(512, 2), (64, 4)])
def test_output_grouping_of_symbolic_masks(TR, G):
    # pre_spgemm's second half: first-fit grouping of the output rows
    rng = np.random.default_rng(TR + G)
    A = rng.random((1024, 256)) < 0.01
    Bm = rng.random((256, 512)) < 0.01
    a, b = W.pack_bits(A), W.pack_bits(Bm)
    cw = ops.symbolic_rows(words_dev(a), 256, words_dev(b), 512)
    g = ops.group_rows(cw, TR, G)
    o = O.group_rows(O.symbolic_rows(a, 256, b, 512), TR, G)
    for k in ("group_id", "group_row", "spill_cnt", "spill_nnz", "spill_rows"):
        assert np.array_equal(g[k].cpu().numpy(), o[k]), k
    assert np.array_equal(words_host(g["group_mask"]), o["group_mask"])


def _int8(rng, M, K):
    A = rng.integers(-128, 128, (M, K), dtype=np.int16).astype(np.int8)
    A[0, : min(K, 4)] = [-128, 127, -1, 0][: min(K, 4)]
    return A


@pytest.mark.parametrize("M,K,N", [(200, 300, 256), (64, 1000, 96), (33, 65, 40), (8, 4096, 512)])
def test_spmm_i8_integer_B_is_exact(M, K, N):
    rng = np.random.default_rng(K)
    A = _int8(rng, M, K)
    B = rng.integers(-8, 9, (K, N)).astype(np.float32)
    C = ops.spmm_i8(dev(A), dev(B)).cpu().numpy()
    assert np.array_equal(C.astype(np.float64), A.astype(np.float64) @ B.astype(np.float64))


@pytest.mark.parametrize("kind", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("M,K,N", [(128, 512, 128), (50, 77, 24), (17, 300, 33)])
def test_bitplane_spmm_matches_oracle(kind, M, K, N):
    rng = np.random.default_rng(M + K + N)
    A = _int8(rng, M, K)
    Bf = rng.standard_normal((K, N), dtype=np.float32)
    tdt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[kind]
    Bt = dev(Bf).to(tdt)
    Bq = Bt.float().cpu().numpy()  # the values the kernel reads
    planes = ops.bitplanes(dev(A.view(np.uint8)), 8)
    C = ops.bitplane_spmm(planes, K, Bt).cpu().numpy()
    C64 = O.bitplane_spmm_f64(A, Bq)
    Cabs = np.abs(A.astype(np.float64)) @ np.abs(Bq.astype(np.float64))
    ms, _, mn = O.rel_errors(C, C64, Cabs)
    assert ms <= 1e-5 and mn <= 1e-5, (ms, mn)
    # the int8 entry point computes the same thing
    C2 = ops.spmm_i8(dev(A), Bt).cpu().numpy()
    assert np.array_equal(C, C2)


def test_unsigned_planes_and_fewer_planes():
    rng = np.random.default_rng(3)
    U = rng.integers(0, 256, (96, 200), dtype=np.int16).astype(np.uint8)
    B = rng.integers(-4, 5, (200, 64)).astype(np.float32)
    planes = ops.bitplanes(dev(U), 8)
    C = ops.bitplane_spmm(planes, 200, dev(B), signed=False).cpu().numpy()
    assert np.array_equal(C.astype(np.float64), U.astype(np.float64) @ B.astype(np.float64))
    # the low 3 planes only: values mod 8
    C3 = ops.bitplane_spmm(planes[:3].contiguous(), 200, dev(B), signed=False).cpu().numpy()
    assert np.array_equal(C3.astype(np.float64), (U % 8).astype(np.float64) @ B.astype(np.float64))


@pytest.mark.parametrize("kind", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("M,K,N,d", [(512, 1024, 256, 0.05), (100, 77, 40, 0.3), (1024, 4096, 512, 0.02)])
def test_int8_planes_along_k(kind, M, K, N, d, monkeypatch):
    # C = [P_0 | ... | P_7] · [w_0 B; ...; w_7 B] through the planned bitmap
    # SpMM, on the tensor cores (BSP_TC=1) and on the CUDA cores (BSP_TC=0)
    rng = np.random.default_rng(M + K + N)
    A = np.where(rng.random((M, K)) < d, rng.integers(-128, 128, (M, K)), 0).astype(np.int8)
    A[0, :3] = [-128, 127, -1]
    Bf = rng.standard_normal((K, N), dtype=np.float32)
    tdt = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[kind]
    Bt = dev(Bf).to(tdt)
    Bq = Bt.float().cpu().numpy()
    C64 = O.bitplane_spmm_f64(A, Bq)
    # error scale of this form: sum_b |w_b| (P_b |B|) — the weighted plane
    # terms it adds (an int8 -1 sets all 8 planes, |weights| summing to 255)
    U = A.view(np.uint8)
    W8 = sum((2.0 ** b) * ((U >> b) & 1).astype(np.float64) for b in range(8))
    Cabs = W8 @ np.abs(Bq.astype(np.float64))
    # the stacked B is exact: block b row k = w_b * B[k]
    Bs = ops.stack_planes_b(Bt, K).float().cpu().numpy()
    Kp = ((K + 31) // 32) * 32
    for b, w in enumerate([1, 2, 4, 8, 16, 32, 64, -128]):
        assert np.array_equal(Bs[b * Kp: b * Kp + K], w * Bq)
        assert not Bs[b * Kp + K: (b + 1) * Kp].any()
    # the plane rows hold the same bits as the plane-major layout
    pr = ops.bitplanes_rows(dev(U)).cpu().numpy().view(np.uint32)
    pm = O.bitplanes(U, 8)
    assert np.array_equal(pr.reshape(M, 8, -1).transpose(1, 0, 2), pm)
    tol = 1e-5 if kind == "f32" else 1e-3
    for tc in ("1", "0"):
        if kind == "f32" and tc == "1":
            continue
        monkeypatch.setenv("BSP_TC", tc)
        mat = ops.Int8Matrix(dev(A))
        C = mat.matmul(Bt).cpu().numpy()
        mat.close()
        ms, _, mn = O.rel_errors(C, C64, Cabs)
        assert ms <= tol, (tc, ms, mn)


@pytest.mark.parametrize("flips", [0.004, 0.03])
@pytest.mark.parametrize("N,pb", [(33, 0.5), (64, 0.01), (2080, 0.02), (4100, 0.3)])
def test_symbolic_planned_counts(N, pb, flips):
    """Delta lists within and past 32 entries, counts of one and of many
    planes, rows without a cluster among clustered ones, rows past the last
    block, odd and even numbers of words: the same bits as without a plan."""
    rng = np.random.default_rng(N)
    M, K = 1003, 2000
    protos = rng.random((3, K)) < 0.1
    bits = protos[rng.integers(0, 3, M)] ^ (rng.random((M, K)) < flips)
    bits[[0, 500, 501, 1002]] = rng.random((4, K)) < 0.1
    bits[700] = False
    a = words_dev(W.pack_bits(bits))
    B = rng.random((K, N)) < pb
    b = words_dev(W.pack_bits(B))
    plan = ops.Plan(a, K, mode=2, min_cluster_rows=8)
    info = plan.info()
    assert info["n_proto"] >= 1 and info["direct_rows"] >= 1
    got = ops.symbolic_rows(a, K, b, N, plan=plan)
    want = W.pack_bits((bits.astype(np.float32) @ B.astype(np.float32)) > 0)
    assert np.array_equal(words_host(got), want)
    assert torch.equal(got, ops.symbolic_rows(a, K, b, N))


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("M,K,N", [(128, 64, 8), (129, 33, 136), (300, 1000, 264), (1000, 3001, 520), (64, 8192, 128),
                                   (5000, 257, 2048), (2400, 5000, 2304)])
def test_int8_values_on_tensor_cores(M, K, N, dt):
    """The product of int8 values kept in the tensor cores' order: every byte
    value, empty tiles, row and column remainders, split reductions, tiled B.
    Integer operands with |sum| <= 4 * 128 * nnz(row) < 2^24: exact in FP32."""
    rng = np.random.default_rng(M + K + N)
    A = (rng.integers(-128, 128, (M, K)) * (rng.random((M, K)) < 0.3)).astype(np.int8)
    A[:, 32:64] = 0
    A[0, :min(K, 256)] = np.arange(-128, 128)[:min(K, 256)]
    B = rng.integers(-4, 5, (K, N))
    mat = ops.Int8Matrix(dev(A))
    assert mat.tiles is not None
    Bt = torch.from_numpy(B).cuda().to(torch.bfloat16 if dt == "bf16" else torch.float16)
    got = mat.matmul(Bt).cpu().numpy()
    out = torch.full((M, N + 8), 7.0, device="cuda")
    mat.matmul(Bt, out=out[:, :N])
    wide = torch.zeros((K, N + 1), dtype=Bt.dtype, device="cuda")  # rows off the 16-byte grid: as planes
    wide[:, :N] = Bt
    planes = mat.matmul(wide[:, :N]).cpu().numpy()
    mat.close()
    want = A.astype(np.float64) @ B.astype(np.float64)
    assert np.array_equal(got, want) and np.array_equal(out[:, :N].cpu().numpy(), want)
    assert (out[:, N:] == 7.0).all() and np.array_equal(planes, want)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N,p", [(256, 256, 16, 0.05), (256, 4096, 256, 0.02), (4096, 1024, 64, 0.03),
                                     (4096, 4096, 256, 0.05), (4096, 4096, 2048, 0.05), (700, 3000, 200, 0.04)])
def test_int8_values_lose_no_precision(M, K, N, p, dt):
    """The values' product, B in two parts, is no further from FP64 than the
    planes' (whose stacked operand is asked for)."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    hit = torch.rand((M, K), device="cuda", generator=g) < p
    v = torch.randint(-128, 128, (M, K), device="cuda", generator=g)
    A = torch.where(hit, v, torch.zeros_like(v)).to(torch.int8)
    B = torch.randn((K, N), device="cuda", generator=g).to(dt)
    m = ops.Int8Matrix(A)
    assert m.tiles is not None
    want = A.double() @ B.double()
    err = lambda C: float((C.double() - want).norm() / want.norm())
    stacked = torch.empty((m.Kc, N), dtype=dt, device="cuda")
    # (errors of 1e-9, where nearly every sum is exact, vary by a few per cent)
    assert err(m.matmul(B)) <= 1.03 * err(m.matmul(B, B_stacked=stacked))
    assert capi.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_int8_values_of_extreme_operands(dt):
    """Infinities, NaN, the largest and the smallest values of B's type through
    its two parts: dense positive A, so that every row holds every column."""
    M, K, N = 200, 96, 40
    rng = np.random.default_rng(6)
    A = rng.integers(1, 128, (M, K)).astype(np.int8)
    fin = torch.finfo(dt)
    B = torch.from_numpy(rng.integers(-8, 9, (K, N)).astype(np.float32)).cuda().to(dt)
    B[3, 1], B[4, 2], B[5, 3] = float("inf"), float("-inf"), float("nan")
    B[:, 4] = 0
    B[7, 4] = fin.max / 256 if dt == torch.bfloat16 else fin.max
    B[:, 5] = 0
    B[8, 5] = fin.tiny * 1.5
    m = ops.Int8Matrix(torch.from_numpy(A).cuda())
    assert m.tiles is not None
    C = m.matmul(B).cpu().numpy()
    want = A.astype(np.float64) @ B.double().cpu().numpy()
    assert np.all(C[:, 1] == np.inf) and np.all(C[:, 2] == -np.inf) and np.all(np.isnan(C[:, 3]))
    rest = [j for j in range(N) if j not in (1, 2, 3)]
    assert np.array_equal(C[:, rest].astype(np.float64), want[:, rest])


@pytest.mark.parametrize("M,K,pad", [(1, 1, 0), (128, 1024, 0), (129, 1025, 0), (300, 2080, 4), (127, 33, 3), (640, 95, 1)])
def test_int8_tile_order(M, K, pad):
    """The values' order and the bit per 128 x 32 tile with a nonzero, at the
    edges of tiles and of blocks, with and without 4-byte rows."""
    import ctypes
    rng = np.random.default_rng(M + K)
    full = rng.integers(-128, 128, (M, K + pad)).astype(np.int8)
    keep = rng.random((-(-M // 128), -(-K // 32))) < 0.5
    full[:, :K] *= keep.repeat(128, 0).repeat(32, 1)[:M, :K]
    A = dev(full)
    n = ctypes.c_size_t()
    capi.call("bsp_i8_tiles_bytes", M, K, ctypes.byref(n))
    tiles = torch.full((n.value,), 77, dtype=torch.int8, device="cuda")
    capi.call("bsp_i8_tiles", A.data_ptr(), M, K, K + pad, tiles.data_ptr(), None)
    got, Kt = tiles.cpu().numpy(), -(-K // 32)
    want = np.zeros((M, Kt * 32), dtype=np.int8)
    want[:, :K] = full[:, :K]
    assert np.array_equal(got[:M * Kt * 32].reshape(Kt, M, 32), want.reshape(M, Kt, 32).transpose(1, 0, 2))
    bits = np.unpackbits(got[M * Kt * 32:].view(np.uint8), bitorder="little").reshape(-(-M // 128), -1)
    hold = np.pad(want, ((0, -M % 128), (0, 0))).reshape(-(-M // 128), 128, Kt, 32).any((1, 3))
    assert np.array_equal(bits[:, :Kt].astype(bool), hold) and not bits[:, Kt:].any()
