"""Workloads of the bitmap SpMM library, through its public entry points.

Each case is one call (or one step) of a program that uses the library: the
plain product, the planned products, a training step, batches, a mask that is
packed and planned anew, the symbolic product and the int8 product.  Inputs
are made on the GPU from the seed alone; what such a program keeps between
calls (packed words, a plan, a batch, an output buffer) is made in prepare().
"""
import math

import torch

from bitwise_spgemm_gb300 import autograd, ops

DEV = "cuda"
DT = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "u8": torch.uint8}
ESZ = {"f32": 4, "bf16": 2, "f16": 2, "u8": 1}

# limits of the drawn cases, from the listed ones
TRAIN_MAX = 4096 * 4096 * 8192        # M*K*N of a 16-bit training step
TRAIN_F32_MAX = 2048 * 2048 * 1024    # ... of an FP32 one
DIRECT_MAX = 2000 * 3001 * 333        # ... of a product without a plan


def listed():
    return [
        # one small layer of an interactive caller: latency
        dict(name="direct_tiny", kind="direct", M=64, K=96, N=16, density=0.1, dtype="f32", values="normal"),
        # the repository's small plain workload: integers, no plan
        dict(name="direct_1024_int", kind="direct", M=1024, K=1024, N=256, density=0.1, dtype="f32", values="int"),
        # sizes that are multiples of nothing
        dict(name="direct_ragged", kind="direct", M=2000, K=3001, N=333, density=0.05, dtype="f32", values="normal"),
        # the headline workload: clustered rows, FP32, a plan that is kept
        dict(name="clustered_f32", kind="clustered", M=8192, K=8192, N=512, protos=64, dtype="f32"),
        # block-structured mask on the tensor cores: the largest forward product
        dict(name="block_bf16", kind="block", M=16384, K=16384, N=2048, density=0.3, dtype="bf16"),
        # training step (forward, gradient of the input, of the mask) in mixed precision
        dict(name="train_bf16", kind="train", M=4096, K=4096, N=8192, density=0.1, dtype="bf16"),
        # the same step in FP32, an ordinary layer
        dict(name="train_f32", kind="train", M=2048, K=2048, N=1024, density=0.1, dtype="f32"),
        # many independent products of mixed sizes in one launch (serving)
        dict(name="batch_bf16", kind="batch", count=512, lo=64, hi=4096, N=128, dtype="bf16"),
        # batched training step: forward, both gradients
        dict(name="batch_train_f16", kind="batch_train", count=128, lo=64, hi=2048, N=96, dtype="f16"),
        # a mask seen for the first time: pack, plan, one product
        dict(name="new_mask_f32", kind="new_mask", M=4096, K=4096, N=256, protos=64, dtype="f32", mask="f32"),
        # pattern of a product of two bitmaps, then the grouping of its rows
        dict(name="symbolic", kind="symbolic", M=8192, K=8192, N=8192, protos=64, b_density=0.002),
        # int8 weights as bit planes, 16-bit activations
        dict(name="int8_bf16", kind="int8", M=4096, K=4096, N=256, density=0.05, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cols(rng, lo, hi):
    """Columns of a dense operand: as often as not a multiple of 8."""
    n = _log(rng, lo, hi)
    return max(8, n // 8 * 8) if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["direct", "direct", "clustered", "block", "train", "train", "batch", "batch_train", "new_mask",
                       "symbolic", "int8"])
    if kind == "direct":
        while True:
            c = dict(kind=kind, M=_log(rng, 32, 4096), K=_log(rng, 32, 4096), N=_cols(rng, 4, 512),
                     density=round(rng.uniform(0.01, 0.2), 4), dtype=rng.choice(["f32", "bf16", "f16"]),
                     values=rng.choice(["int", "normal"]))
            if c["M"] * c["K"] * c["N"] <= DIRECT_MAX and c["density"] * c["M"] * c["K"] * c["N"] <= 0.05 * DIRECT_MAX:
                return c
    if kind == "clustered":
        return dict(kind=kind, M=_log(rng, 512, 8192), K=_log(rng, 512, 8192), N=_cols(rng, 32, 512),
                    protos=_log(rng, 8, 64), dtype=rng.choice(["f32", "bf16", "f16"]))
    if kind == "block":
        return dict(kind=kind, M=_log(rng, 1024, 16384), K=_log(rng, 1024, 16384), N=_cols(rng, 64, 1024),
                    density=round(rng.uniform(0.05, 0.3), 4), dtype=rng.choice(["bf16", "f16"]))
    if kind == "train":
        dt = rng.choice(["bf16", "f16", "f32"])
        while True:
            c = dict(kind=kind, M=_log(rng, 256, 4096), K=_log(rng, 256, 4096), N=_log(rng, 64, 8192) // 8 * 8,
                     density=round(rng.uniform(0.05, 0.1), 4), dtype=dt)
            if c["M"] * c["K"] * c["N"] <= (TRAIN_F32_MAX if dt == "f32" else TRAIN_MAX):
                return c
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 16, 512), lo=64, hi=_log(rng, 256, 4096), N=_log(rng, 16, 128) // 8 * 8,
                    dtype=rng.choice(["bf16", "f16"]))
    if kind == "batch_train":
        return dict(kind=kind, count=_log(rng, 8, 128), lo=64, hi=_log(rng, 256, 2048), N=_log(rng, 16, 128) // 8 * 8,
                    dtype=rng.choice(["bf16", "f16"]))
    if kind == "new_mask":
        return dict(kind=kind, M=_log(rng, 256, 4096), K=_log(rng, 256, 4096), N=_cols(rng, 32, 256),
                    protos=_log(rng, 8, 64), dtype=rng.choice(["f32", "bf16"]), mask=rng.choice(["f32", "bf16", "u8"]))
    if kind == "symbolic":
        return dict(kind=kind, M=_log(rng, 512, 8192), K=_log(rng, 512, 8192), N=_log(rng, 512, 8192),
                    protos=_log(rng, 8, 64), b_density=round(rng.uniform(0.0005, 0.002), 5))
    return dict(kind=kind, M=_log(rng, 256, 4096), K=_log(rng, 256, 4096), N=_log(rng, 16, 256) // 8 * 8,
                density=round(rng.uniform(0.02, 0.05), 4), dtype=rng.choice(["bf16", "f16"]))


# ---- inputs (plain torch, from the seed alone) ---------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _bits(g, rows, cols, p):
    return torch.rand((rows, cols), device=DEV, generator=g) < p


def _clustered(g, M, K, protos):
    """Rows are copies of a few random prototypes with independent bit flips."""
    p = _bits(g, protos, K, 0.05)
    idx = torch.randint(protos, (M,), device=DEV, generator=g)
    return p[idx] ^ _bits(g, M, K, 0.002)


def _blocks(g, M, K, p):
    """32x32 blocks present with probability p, dense inside."""
    t = _bits(g, (M + 31) // 32, (K + 31) // 32, p)
    t = t.repeat_interleave(32, 0)[:M].repeat_interleave(32, 1)[:, :K]
    return t & _bits(g, M, K, 0.8)


def _dense(g, rows, cols, dtype, values="normal"):
    if values == "int":
        return torch.randint(-8, 9, (rows, cols), device=DEV, generator=g).to(DT[dtype])
    return torch.randn((rows, cols), device=DEV, generator=g).to(DT[dtype])


def _mask(case, g):
    k = case["kind"]
    if k in ("direct", "train"):
        return _bits(g, case["M"], case["K"], case["density"])
    if k == "block":
        return _blocks(g, case["M"], case["K"], case["density"])
    return _clustered(g, case["M"], case["K"], case["protos"])


def _sizes(case):
    """The sizes of a batch's problems: the same for every seed."""
    import random
    r = random.Random(7)
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [(32 * max(1, round(math.exp(r.uniform(lo, hi)) / 32)), 32 * max(1, round(math.exp(r.uniform(lo, hi)) / 32)),
             r.uniform(0.01, 0.3)) for _ in range(case["count"])]


def _batch_inputs(case, seed):
    g = _gen(seed)
    N, dt = case["N"], case["dtype"]
    got = []
    for M, K, d in _sizes(case):
        A = _bits(g, M, K, d)
        X = _dense(g, K, N, dt)
        got.append((A, X, _dense(g, M, N, dt) if case["kind"] == "batch_train" else None))
    return got


def _int8(case, g):
    hit = _bits(g, case["M"], case["K"], case["density"])
    v = torch.randint(-128, 127, hit.shape, device=DEV, generator=g)
    return torch.where(hit, v + (v >= 0).long(), torch.zeros_like(v)).to(torch.int8)


# ---- the cases -------------------------------------------------------------------

def prepare(case, seed):
    k = case["kind"]
    s = dict(kind=k)
    if k in ("batch", "batch_train"):
        N = case["N"]
        probs = _batch_inputs(case, seed)
        rows = sum(A.shape[0] for A, _, _ in probs)
        Y = torch.empty((rows, N), device=DEV)
        words, fwd, r0 = [], [], 0
        for A, X, _ in probs:
            w = ops.pack_rows(A.to(torch.uint8))
            words.append(w)
            fwd.append((w, A.shape[1], X, Y[r0:r0 + A.shape[0]]))
            r0 += A.shape[0]
        s.update(batch=ops.Batch(fwd), Y=Y)
        if k == "batch_train":
            dX = torch.empty((sum(A.shape[1] for A, _, _ in probs), N), device=DEV)
            dA = torch.empty(sum(A.numel() for A, _, _ in probs), device=DEV)
            bwd, x0, a0 = [], 0, 0
            for w, (A, X, G) in zip(words, probs):
                M, K = A.shape
                bwd.append((w, K, X, G, dX[x0:x0 + K], dA[a0:a0 + M * K].view(M, K)))
                x0, a0 = x0 + K, a0 + M * K
            s.update(grad=ops.BatchGrad(bwd), dX=dX, dA=dA)
        return s
    g = _gen(seed)
    if k == "int8":
        s["A"] = ops.Int8Matrix(_int8(case, g))
        s["B"] = _dense(g, case["K"], case["N"], case["dtype"])
        return s
    A = _mask(case, g)
    if k == "new_mask":
        s.update(mask=A.to(DT[case["mask"]]), K=case["K"], B=_dense(g, case["K"], case["N"], case["dtype"]))
        return s
    if k == "train":
        X = _dense(g, case["K"], case["N"], case["dtype"])
        # the gradient of a 16-bit layer above, in FP32 as the output is
        G = _dense(g, case["M"], case["N"], case["dtype"]).float()
        plan = ops.Plan(ops.pack_rows(A.to(torch.uint8)), case["K"])
        s.update(mask=A.float().requires_grad_(), X=X.requires_grad_(), G=G, plan=plan)
        return s
    s.update(words=ops.pack_rows(A.to(torch.uint8)), K=case["K"])
    if k == "symbolic":
        s.update(b_words=ops.pack_rows(_bits(g, case["K"], case["N"], case["b_density"]).to(torch.uint8)), N=case["N"],
                 plan=ops.Plan(s["words"], case["K"]))
        return s
    s.update(B=_dense(g, case["K"], case["N"], case["dtype"], case.get("values", "normal")), plan=None,
             out=torch.empty((case["M"], case["N"]), device=DEV))
    if k != "direct":
        s["plan"] = ops.Plan(s["words"], case["K"])
        s["workspace"] = torch.empty(max(1, s["plan"].workspace_bytes(case["N"])), dtype=torch.uint8, device=DEV)
    return s


def run(s):
    k = s["kind"]
    if k == "batch":
        s["batch"].run()
        return {"Y": s["Y"]}
    if k == "batch_train":
        s["batch"].run()
        s["grad"].run()
        return {"Y": s["Y"], "dX": s["dX"], "dA": s["dA"]}
    if k == "int8":
        return {"C": s["A"].matmul(s["B"])}
    if k == "new_mask":
        words = ops.pack_rows(s["mask"])
        plan = ops.Plan(words, s["K"])
        C = ops.spmm(words, s["K"], s["B"], plan=plan)
        plan.close_async()
        return {"C": C, "words": words}
    if k == "train":
        Y = autograd.bitmap_matmul(s["mask"], s["X"], plan=s["plan"])
        dA, dX = torch.autograd.grad(Y, (s["mask"], s["X"]), s["G"])
        return {"Y": Y, "dX": dX, "dA": dA}
    if k == "symbolic":
        c = ops.symbolic_rows(s["words"], s["K"], s["b_words"], s["N"], plan=s["plan"])
        return dict(ops.group_rows(c, 512, 2), mask=c)
    return {"C": ops.spmm(s["words"], s["K"], s["B"], plan=s["plan"], out=s["out"], workspace=s.get("workspace"))}


def _nnz(case):
    M, K = case["M"], case["K"]
    k = case["kind"]
    if k in ("direct", "train"):
        return M * K * case["density"]
    if k == "block":
        return M * K * case["density"] * 0.8
    return M * K * 0.05


def work(case):
    """Inputs read once, outputs written once; one multiply-add per set bit
    (nonzero value) and column, and for the mask's gradient too."""
    k = case["kind"]
    if k in ("batch", "batch_train"):
        N, b, f = case["N"], 0, 0
        for M, K, d in _sizes(case):
            step = 2 * M * K * d * N
            b += M * K / 8 + K * N * 2 + M * N * 4
            f += step
            if k == "batch_train":  # G too, dX, dA
                b += M * N * 2 + K * N * 4 + M * K * 4
                f += 2 * step
        return {"bytes": b, "flops": f}
    M, K, N = case["M"], case["K"], case["N"]
    e = ESZ[case["dtype"]] if "dtype" in case else 0
    bits = M * ((K + 31) // 32) * 4
    if k == "train":  # mask, X and G in; Y, dX and dA out
        return {"bytes": M * K * 4 + K * N * e + M * N * 4 + M * N * 4 + K * N * e + M * K * 4, "flops": 3 * 2 * _nnz(case) * N}
    if k == "new_mask":
        return {"bytes": M * K * ESZ[case["mask"]] + bits + K * N * e + M * N * 4, "flops": 2 * _nnz(case) * N}
    if k == "symbolic":
        nw = (N + 31) // 32
        tiles = (M + 511) // 512 * nw
        out = M * nw * 8 + tiles * (2 * 4 + 2 * 32 * 4 + 8 + 512 * 4) + 8
        return {"bytes": bits + K * nw * 4 + out, "flops": 0}
    if k == "int8":
        return {"bytes": M * K + K * N * e + M * N * 4, "flops": 2 * M * K * case["density"] * N}
    return {"bytes": bits + K * N * e + M * N * 4, "flops": 2 * _nnz(case) * N}


def exact(case, seed):
    k = case["kind"]
    if k == "symbolic":
        return None  # whole numbers only
    if k in ("batch", "batch_train"):
        Y, dX, dA = [], [], []
        for A, X, G in _batch_inputs(case, seed):
            Ad, Xd = A.double(), X.double()
            Y.append(Ad @ Xd)
            if G is not None:
                dX.append(Ad.T @ G.double())
                dA.append(((G.double() @ Xd.T) * Ad).reshape(-1))
        got = {"Y": torch.cat(Y)}
        if k == "batch_train":
            got.update(dX=torch.cat(dX), dA=torch.cat(dA))
        return got
    g = _gen(seed)
    if k == "int8":
        A = _int8(case, g).double()
        return {"C": A @ _dense(g, case["K"], case["N"], case["dtype"]).double()}
    A = _mask(case, g).double()
    if k == "train":
        X = _dense(g, case["K"], case["N"], case["dtype"]).double()
        G = _dense(g, case["M"], case["N"], case["dtype"]).double()
        return {"Y": A @ X, "dX": A.T @ G, "dA": (G @ X.T) * A}
    C = A @ _dense(g, case["K"], case["N"], case["dtype"], case.get("values", "normal")).double()
    return {"C": C, "words": None} if k == "new_mask" else {"C": C}
