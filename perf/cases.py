"""The work that a program has this library do, as cases that can be timed.

Every case goes through the public entry points of ``tensor_bf_main_gb300``: the exact
epsilon self-join in its arithmetics (plain FP64, FP16 / BF16, BF16 hi+lo, FP8), with and
without learned pruning, from host, page-locked and device memory; the reference's driver
call; neighbour lists; the join of two point sets; the count of given rows on the exact
arbiter; and the training of a projection.  The data have the shapes and distributions of
the benchmark configurations (``tensor_bf_main_gb300/datagen.py``), made on the GPU from
the seed; a radius is calibrated for a mean number of neighbours, as the benchmark does.
"""
import ctypes
import math

import numpy as np
import torch

import tensor_bf_main_gb300 as ej

DEV = "cuda:0"


def listed():
    return [
        # a script's first call: a sample-sized set in a numpy array, nothing but defaults
        dict(name="sample_host", op="self_join", kind="uniform", n=1000, d=18, target=8,
             precision="auto", k=0, where="host", keep=False),
        # the reference's driver call (its tensor-core search mode) on its padded host array
        dict(name="driver_host", op="driver", kind="gmm", n=25_013, d=18, target=32, mode=4),
        # the plain FP64 tensor-core join, 10,000 x 128 uniform
        dict(name="plain_fp64", op="self_join", kind="uniform", n=10_000, d=128, target=32,
             precision="fp64_dmma", k=0, where="device", keep=True),
        # sampled rows of a large set recounted on the exact FP64 arbiter
        dict(name="arbiter_rows", op="query", kind="gmm", n=200_003, d=64, target=64, nq=500),
        # the plain join at scale in FP16: 1M x 128, 64 Gaussians
        dict(name="dense_fp16", op="self_join", kind="gmm", n=1_000_000, d=128, target=64,
             precision="fp16", k=0, where="device", keep=True),
        # power-law spectrum, offset data, BF16 hi+lo, d = 256
        dict(name="dense_split", op="self_join", kind="powerlaw", n=500_000, d=256, target=128,
             precision="bf16_split", k=0, where="device", keep=True),
        # the benchmark's default: learned pruning at 4M x 64, BF16 hi+lo
        dict(name="pruned_split", op="self_join", kind="latent", n=4_000_000, d=64, target=50,
             precision="bf16_split", k=8, where="device", keep=True),
        # high dimension in FP8 with a k = 16 projection
        dict(name="sphere_fp8", op="self_join", kind="sphere", n=250_007, d=1024, target=20,
             precision="fp8_e4m3", k=16, where="device", keep=True),
        # end to end from page-locked host memory, training overlapped with the copy
        dict(name="pinned_pruned", op="self_join", kind="latent", n=1_000_003, d=64, target=50,
             precision="auto", k=8, where="pinned", keep=True),
        # neighbour lists of a mid-sized set through the C ABI, into buffers that the program keeps
        dict(name="lists", op="lists", kind="gmm", n=150_011, d=64, target=32, precision="auto",
             k=0, where="device", keep=False),
        # two point sets of an odd dimension, BF16 (what AUTO takes beyond d = 128)
        dict(name="cross_bf16", op="cross", kind="gmm", n=300_007, d=200, target=32, nq=40_001,
             precision="auto", keep=False),
        # a projection trained once, to be saved and reused
        dict(name="train", op="train", kind="latent", n=1_000_000, d=64, target=50, k=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng, d, most_pairs_d, lo, hi):
    """A number of points whose n^2 d stays below most_pairs_d."""
    return _log(rng, lo, max(lo + 1, min(hi, int(math.sqrt(most_pairs_d / d)))))


def draw(rng):
    op = rng.choice(["small", "small", "dense", "dense", "dense", "pruned", "pruned", "fp64",
                     "lists", "cross", "query", "driver", "train"])
    dense_kinds = ["uniform", "gmm", "powerlaw"]
    precisions = ["auto", "fp16", "bf16", "bf16_split", "fp8_e4m3"]
    target = _log(rng, 4, 128)
    if op == "small":
        return dict(op="self_join", kind=rng.choice(dense_kinds), n=_log(rng, 100, 20_000),
                    d=_log(rng, 2, 256), target=target, precision=rng.choice(precisions), k=0,
                    where=rng.choice(["host", "device"]), keep=rng.random() < 0.5)
    if op == "dense":
        d = _log(rng, 16, 1024)
        return dict(op="self_join", kind=rng.choice(dense_kinds), n=_rows(rng, d, 5e13, 20_000, 1_000_000),
                    d=d, target=target, precision=rng.choice(precisions), k=0, where="device",
                    keep=rng.random() < 0.5)
    if op == "pruned":
        kind = rng.choice(["latent", "latent", "sphere"])
        d = _log(rng, 16, 128) if kind == "latent" else _log(rng, 256, 1024)
        n = _log(rng, 50_000, 3_000_000) if kind == "latent" else _rows(rng, d, 6e13, 20_000, 400_000)
        return dict(op="self_join", kind=kind, n=n, d=d, target=target,
                    precision=rng.choice(["auto", "bf16", "bf16_split", "fp8_e4m3"]),
                    k=rng.choice([8, 16]), where=rng.choice(["device", "device", "pinned"]),
                    keep=rng.random() < 0.5)
    if op == "fp64":
        d = _log(rng, 3, 256)
        return dict(op="self_join", kind=rng.choice(dense_kinds), n=_rows(rng, d, 5e10, 300, 40_000),
                    d=d, target=target, precision=rng.choice(["fp64_dmma", "fp64_direct"]), k=0,
                    where=rng.choice(["host", "device"]), keep=rng.random() < 0.5)
    if op == "lists":
        return dict(op="lists", kind=rng.choice(dense_kinds), n=_log(rng, 500, 300_000),
                    d=_log(rng, 3, 128), target=_log(rng, 4, 64), precision=rng.choice(precisions[:4]),
                    k=0, where=rng.choice(["host", "device"]), keep=False)
    if op == "cross":
        return dict(op="cross", kind=rng.choice(dense_kinds), n=_log(rng, 1_000, 500_000),
                    d=_log(rng, 3, 400), target=target, nq=_log(rng, 10, 50_000),
                    precision=rng.choice(precisions), keep=False)
    if op == "query":
        return dict(op="query", kind=rng.choice(dense_kinds), n=_log(rng, 1_000, 300_000),
                    d=_log(rng, 3, 128), target=target, nq=_log(rng, 1, 700))
    if op == "driver":
        return dict(op="driver", kind=rng.choice(dense_kinds), n=_log(rng, 500, 60_000),
                    d=_log(rng, 2, 128), target=target, mode=rng.choice([3, 4]))
    return dict(op="train", kind="latent", n=_log(rng, 20_000, 2_000_000), d=_log(rng, 16, 128),
                target=target, k=rng.choice([8, 16]))


# ---------------------------------------------------------------- inputs --

def _points(kind, n, d, gen, cgen):
    """n x d float64 on the GPU; cgen (a CPU generator) makes what the rows share: centres,
    rotations, embeddings."""
    def randn(*s):
        return torch.randn(*s, generator=gen, device=DEV, dtype=torch.float64)

    if kind == "uniform":
        return torch.rand(n, d, generator=gen, device=DEV, dtype=torch.float64)
    if kind == "gmm":
        centres = torch.rand(64, d, generator=cgen, dtype=torch.float64).to(DEV)
        lab = torch.randint(0, 64, (n,), generator=gen, device=DEV)
        return randn(n, d).mul_(0.05).add_(centres[lab])
    if kind == "powerlaw":
        q, r = torch.linalg.qr(torch.randn(d, d, generator=cgen, dtype=torch.float64))
        lam = torch.arange(1, d + 1, dtype=torch.float64) ** -0.75
        m = ((q * torch.sign(torch.diagonal(r))) * lam).T.contiguous().to(DEV)
        return (randn(n, d) @ m).add_(10.0)
    if kind == "latent":
        centres = torch.rand(256, 8, generator=cgen, dtype=torch.float64).to(DEV)
        e = torch.linalg.qr(torch.randn(d, 8, generator=cgen, dtype=torch.float64))[0].to(DEV)
        lab = torch.randint(0, 256, (n,), generator=gen, device=DEV)
        z = randn(n, 8).mul_(0.02).add_(centres[lab])
        return randn(n, d).mul_(0.01).add_(z @ e.T)
    centres = torch.randn(1000, d, generator=cgen, dtype=torch.float64)
    centres = (centres / centres.norm(dim=1, keepdim=True)).to(DEV)
    lab = torch.randint(0, 1000, (n,), generator=gen, device=DEV)
    x = randn(n, d).mul_(0.016573473373427988 * math.sqrt(1024.0 / d)).add_(centres[lab])
    return x.div_(x.norm(dim=1, keepdim=True))


def _radius(x, target, queries=None):
    """The radius with about `target` neighbours a row (pooled nearest distances of 32 rows),
    to four digits."""
    src = x if queries is None else queries
    q = src[torch.linspace(0, src.shape[0] - 1, min(32, src.shape[0]), dtype=torch.float64).long().to(DEV)]
    mu = x[: 1 << 16].mean(0)
    q = q - mu
    want = max(1, min(int(target), x.shape[0])) * q.shape[0]
    best = None
    for lo in range(0, x.shape[0], 1 << 17):
        c = x[lo:lo + (1 << 17)] - mu
        d2 = (q * q).sum(1)[:, None] + (c * c).sum(1)[None, :] - 2.0 * (q @ c.T)
        d2 = d2.reshape(-1)
        d2 = torch.topk(d2, min(want, d2.numel()), largest=False).values
        best = d2 if best is None else torch.cat([best, d2])
        best = torch.topk(best, min(want, best.numel()), largest=False).values
    return float("%.4g" % math.sqrt(max(float(best.max()), 1e-12)))


def _gens(seed):
    return (torch.Generator(device=DEV).manual_seed(seed),
            torch.Generator().manual_seed(seed + 1))


def prepare(case, seed):
    gen, cgen = _gens(seed)
    n, d, op = case["n"], case["d"], case["op"]
    x = _points(case["kind"], n, d, gen, cgen)
    s = {"case": case, "q": None}
    if op == "cross":
        # both sets from one distribution: the queries are further rows of it
        cgen = _gens(seed)[1]
        s["q"] = _points(case["kind"], case["nq"], d, gen, cgen)
    s["eps"] = _radius(x, case["target"], s["q"])
    if op == "query":
        s["rows"] = np.sort(np.random.RandomState(seed % (1 << 32)).choice(n, case["nq"] if case["nq"] < n else n,
                                                                           replace=False)).astype(np.uint64)
    where = case.get("where", "host" if op == "driver" else "device")
    if op == "driver":
        # the reference's layout: rows padded to a multiple of 16 columns, 15 zero rows behind
        cd = (d + 15) // 16 * 16
        a = np.zeros((n + 15, cd), dtype=np.float64)
        a[:n, :d] = x.cpu().numpy()
        s["x"], s["cd"] = a.reshape(-1), cd
    elif where == "host":
        s["x"] = x.cpu().numpy()
    elif where == "pinned":
        s["x"] = torch.empty(n, d, dtype=torch.float64, pin_memory=True).copy_(x)
    else:
        s["x"] = x
    if op == "self_join":
        # device callers receive the counts on the device, host callers on the host
        s["out"] = torch.empty(n, dtype=torch.int32, device=DEV) if where == "device" else True
    if op == "lists":
        # buffers where the points are, with room for twice the expected neighbours
        dev = DEV if where == "device" else "cpu"
        s["x"] = torch.as_tensor(s["x"])
        s["offsets"] = torch.zeros(n + 1, dtype=torch.int64, device=dev)
        s["neighbors"] = torch.zeros(2 * n * case["target"] + 1024, dtype=torch.int32, device=dev)
        opt = ej.Options()
        ej.load_library().ejoin_default_options(ctypes.byref(opt))
        opt.precision = ej.Precision.parse(case["precision"])
        s["opt"] = opt
    return s


# ------------------------------------------------------------------ pass --

def run(s):
    c = s["case"]
    op, x, eps = c["op"], s["x"], s["eps"]
    if op == "self_join":
        counts, total, _ = ej.self_join(x, eps, precision=c["precision"], proj_k=c["k"],
                                        counts=s["out"], keep_scratch=c["keep"])
        return counts, total
    if op == "driver":
        return ej.GPUJoinMainBruteForce(c["mode"], 0, x, c["n"], eps, c["d"], s["cd"])
    if op == "lists":
        total = ctypes.c_uint64(0)
        st = ej.load_library().ejoin_neighbor_lists(
            x.data_ptr(), c["n"], c["d"], eps, ctypes.byref(s["opt"]), s["offsets"].data_ptr(),
            s["neighbors"].data_ptr(), s["neighbors"].numel(), ctypes.byref(total), None)
        if st:
            raise RuntimeError("ejoin_neighbor_lists: status %d" % st)
        return s["offsets"], s["neighbors"], total.value
    if op == "cross":
        counts, total, _ = ej.join_counts(s["q"], x, eps, precision=c["precision"])
        return counts, total
    if op == "query":
        return ej.query_counts(x, eps, s["rows"])
    p, sigma, _ = ej.train_projection(x, eps, k=c["k"])
    return p, sigma


def work(case):
    n, d, op = case["n"], case["d"], case["op"]
    if op == "cross":
        return {"bytes": 8.0 * d * (n + case["nq"]) + 4.0 * case["nq"], "flops": 2.0 * d * n * case["nq"]}
    if op == "query":
        return {"bytes": 8.0 * d * n + 12.0 * case["nq"], "flops": 3.0 * d * n * case["nq"]}
    if op == "train":
        # 50 steps over minibatches of 65,536 sampled pairs, forward and backward, after one
        # read of the points
        return {"bytes": 8.0 * d * n, "flops": 50.0 * 65536 * 4.0 * case["k"] * d}
    pairs = n * (n + 1) / 2.0
    if case.get("k") and case["kind"] == "latent":
        pairs /= 256.0  # the pairs within the clusters
    per_pair = {"fp64_direct": 3.0, "bf16_split": 6.0}.get(case.get("precision"), 2.0) * d
    out = 4.0 * n
    if op == "driver":
        out = 8.0
    if op == "lists":
        out = 8.0 * (n + 1) + 4.0 * n * case["target"]
    return {"bytes": 8.0 * d * n + out, "flops": per_pair * pairs}


# ----------------------------------------------------------------- exact --

def _count(q, x, eps):
    """Neighbours of each row of q among x, by differences in float64."""
    out = torch.empty(q.shape[0], dtype=torch.int64, device=DEV)
    step = max(1, int(2e8 // (x.shape[0] * x.shape[1])))
    for lo in range(0, q.shape[0], step):
        t = q[lo:lo + step, None, :] - x[None, :, :]
        out[lo:lo + step] = (t.mul_(t).sum(2).sqrt_() <= eps).sum(1)
    return out


def exact(case, seed):
    n, d, op = case["n"], case["d"], case["op"]
    rows = case.get("nq", n)
    if op in ("train", "lists") or float(rows) * n * d > 3e10:
        return None
    s = prepare(case, seed)
    x = s["x"]
    if op == "driver":
        x = x.reshape(n + 15, s["cd"])[:n, :d].copy()
    x = torch.as_tensor(x).to(DEV)
    q = s["q"] if op == "cross" else x[torch.from_numpy(s["rows"].astype(np.int64)).to(DEV)] if op == "query" else x
    counts = _count(q, x, s["eps"])
    total = int(counts.sum())
    counts = counts.to(torch.int32)
    return total if op == "driver" else counts.cpu().numpy() if op == "query" else (counts, total)
