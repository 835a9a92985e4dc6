"""The work that users of this package have it do, as measurable cases.

A case is a flat dict.  `op` names the operator:

  cdist    kermac.cdist(a, b, p=..., skip_epilogue=...)
  kernel   kermac.run_kernel(descriptor, a, b, bandwidth=..., ...): a materialised kernel matrix
  grad     kermac.cdist_grad(a, b, c, d, p=...)
  matvec   kermac.kernel_matvec(descriptor, a, b, c, bandwidth=...): the kernel matrix is never stored

`layout` says how the caller holds its points: "rows" is torch's own layout (one point per
contiguous row, results allocated by the call), "cols" the transposed storage a[K, M], b[K, N]
with an output buffer that is kept between calls.  `sample` is the distribution of the points.
"""
import math

import torch

import kermac_b200 as kermac

GAUSSIAN_L2 = kermac.KernelDescriptor(kermac.InnerOperator.DIFF, kermac.PowerType.SQUARE,
                                      kermac.PowerType.NOOP, kermac.KernelType.GAUSSIAN)
DESCRIPTORS = {
    "laplace_l1": kermac.kernel_descriptor_laplace_l1,
    "laplace_l2": kermac.kernel_descriptor_laplace_l2,
    "gaussian": GAUSSIAN_L2,
}


def listed():
    return [
        # A handful of points against a handful of centres inside a training loop: nothing but the
        # cost of a call.
        dict(name="cdist_tiny_rows", op="cdist", L=1, M=128, N=96, K=10, p=2.0, layout="rows", sample="normal"),
        # The small problem of the benchmark (unit-cube features, Euclidean), called back to back.
        dict(name="cdist_small", op="cdist", L=1, M=2048, N=2048, K=64, p=2.0, layout="cols", sample="uniform"),
        # A batch of two mid-size problems straight from torch tensors, the shape the tests check.
        dict(name="cdist_batch_rows", op="cdist", L=2, M=1000, N=1000, K=64, p=1.0, layout="rows", sample="normal"),
        # The headline problem: Manhattan distances of 30000 x 30000 embeddings of 1024 features.
        dict(name="cdist_large_l1", op="cdist", L=1, M=30000, N=30000, K=1024, p=1.0, layout="cols", sample="normal"),
        # Euclidean distances of a large data set held as torch rows, odd extents.
        dict(name="cdist_large_l2_rows", op="cdist", L=1, M=20011, N=15013, K=512, p=2.0, layout="rows",
             sample="normal"),
        # Fractional order, four data sets against one broadcast set of centres.
        dict(name="cdist_batch_frac", op="cdist", L=4, M=16384, N=16384, K=512, p=1.3, layout="cols",
             sample="symmetric", broadcast_b=True),
        # Fitting a kernel method: K(X, X) + lambda I of a tabular data set for a solver.
        dict(name="kernel_fit_rows", op="kernel", L=1, M=8000, N=8000, K=96, kernel="laplace_l2", layout="rows",
             sample="normal", same=True, bandwidth=10.0, regularization=1e-3),
        # Gradient of a kernel model with a few outputs: a long sum over training points.
        dict(name="grad_long", op="grad", L=1, K=30000, M=4096, N=256, O=4, p=1.0),
        # Gradient of a small model, the shape the tests check, sixteen outputs.
        dict(name="grad_small", op="grad", L=1, K=64, M=1000, N=1000, O=16, p=1.5),
        # Gradient of a many-output model.
        dict(name="grad_wide", op="grad", L=1, K=30000, M=4096, N=256, O=32, p=1.0),
        # One step of an iterative solver over a kernel matrix that is too large to keep around.
        dict(name="matvec_large", op="matvec", L=1, M=131072, N=65536, K=64, O=16, kernel="laplace_l2",
             layout="cols", sample="normal", bandwidth=8.0),
        # Prediction: a thousand new points against a fitted model, torch rows of an odd width.
        dict(name="matvec_predict_rows", op="matvec", L=1, M=10007, N=1009, K=27, O=5, kernel="laplace_l2",
             layout="rows", sample="normal", bandwidth=8.0),
    ]


# ------------------------------------------------------------------------------------ drawing
def _log_int(rng, low, high):
    """An integer spread evenly over the logarithm of [low, high]; every second one a multiple of 8."""
    v = math.exp(rng.uniform(math.log(low), math.log(high + 1)))
    v = min(high, max(low, int(v)))
    if rng.random() < 0.5 and v >= 16:
        v -= v % 8
    return v


def _cost(case):
    """Arithmetic of a case in FP32 operations, fractional powers weighted by what they take."""
    frac = 5.0 if case.get("p", 2.0) not in (1.0, 2.0) else 1.0
    pairs = float(case["L"]) * case["M"] * case["N"]
    if case["op"] == "grad":
        return pairs * case["K"] * (2 * frac + case["O"])
    if case["op"] == "matvec":
        return pairs * (2 * case["K"] * frac + 2 * case["O"] + 20)
    return pairs * (2 * case["K"] * frac + 20)


_COST_LIMIT = 3.0e12       # the largest listed case: 5.5e12
_OUT_LIMIT = 4.0e8         # elements of a result


def _out_elements(case):
    if case["op"] == "matvec":
        return case["L"] * case["N"] * case["O"]
    return case["L"] * case["M"] * case["N"] * case.get("O", 1)


def _bandwidth(rng, kernel, K):
    """A width of about the distance between two points, as the median heuristic gives it."""
    typical = 1.13 * K if kernel == "laplace_l1" else math.sqrt(2.0 * K)
    return round(typical * rng.choice((0.5, 1.0)), 3)


def _draw_one(rng):
    op = rng.choice(("cdist", "cdist", "kernel", "grad", "matvec"))
    if op == "grad":
        return dict(op=op, L=rng.choice((1, 1, 1, 2)), K=_log_int(rng, 64, 30000), M=_log_int(rng, 64, 4096),
                    N=_log_int(rng, 16, 1000), O=_log_int(rng, 1, 64),
                    p=rng.choice((1.0, 1.5, 2.0, round(rng.uniform(1.1, 2.9), 1))))
    common = dict(op=op, layout=rng.choice(("rows", "cols")), sample=rng.choice(("normal", "uniform", "symmetric")))
    if op == "cdist":
        return dict(common, L=rng.choice((1, 1, 2, 4)), M=_log_int(rng, 64, 30000), N=_log_int(rng, 64, 30000),
                    K=_log_int(rng, 8, 1024), p=rng.choice((1.0, 2.0, 1.3, round(rng.uniform(1.1, 2.9), 1))),
                    broadcast_b=rng.random() < 0.3, skip_epilogue=rng.random() < 0.2)
    kernel = rng.choice(("laplace_l1", "laplace_l2", "gaussian"))
    if op == "kernel":
        same = rng.random() < 0.5
        M, K = _log_int(rng, 64, 20000), _log_int(rng, 8, 1024)
        return dict(common, L=rng.choice((1, 1, 2)), M=M, N=M if same else _log_int(rng, 64, 20000), K=K, kernel=kernel,
                    same=same, bandwidth=_bandwidth(rng, kernel, K), regularization=1e-3 if same else 0.0,
                    tensor_bandwidth=rng.random() < 0.3)
    K = _log_int(rng, 8, 512)
    return dict(common, L=1, M=_log_int(rng, 500, 131072), N=_log_int(rng, 64, 131072), K=K, O=_log_int(rng, 1, 32),
                kernel=kernel, bandwidth=_bandwidth(rng, kernel, K))


def draw(rng):
    """One more case of the same ranges; none costs more than the largest listed one."""
    while True:
        case = _draw_one(rng)
        if _cost(case) <= _COST_LIMIT and _out_elements(case) <= _OUT_LIMIT:
            return case


# ------------------------------------------------------------------------------------ inputs
def _points(gen, case, L, count):
    """`count` points of K features, shape (count, K) or (L, count, K), in the case's layout."""
    shape = (count, case["K"]) if L == 1 else (L, count, case["K"])
    if case["layout"] == "cols":
        shape = shape[:-2] + (shape[-1], shape[-2])
    if case["sample"] == "normal":
        x = torch.randn(shape, generator=gen, device="cuda")
    else:
        x = torch.rand(shape, generator=gen, device="cuda")
        if case["sample"] == "symmetric":
            x.mul_(2.0).sub_(1.0)
    return x.transpose(-1, -2) if case["layout"] == "cols" else x


def _out_buffer(case, L, rows, cols):
    """The kept output buffer of a "cols" caller: out[N, M] storage seen as (M, N)."""
    if case["layout"] != "cols":
        return None
    shape = (cols, rows) if L == 1 else (L, cols, rows)
    return torch.empty(shape, device="cuda").transpose(-1, -2)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op, L = case["op"], case["L"]
    state = dict(op=op)
    if op == "grad":
        lead = () if L == 1 else (L,)
        K, M, N, O = case["K"], case["M"], case["N"], case["O"]
        # weights are kernel values, the rest is standardised data
        state["a"] = torch.rand(lead + (K, M), generator=gen, device="cuda")
        state["b"] = torch.randn(lead + (N, K), generator=gen, device="cuda")
        state["c"] = torch.randn(lead + (O, K), generator=gen, device="cuda")
        state["d"] = torch.randn(lead + (N, M), generator=gen, device="cuda")
        state["p"] = case["p"]
        return state
    state["a"] = _points(gen, case, L, case["M"])
    if case.get("same"):
        state["b"] = state["a"]
    else:
        state["b"] = _points(gen, case, 1 if case.get("broadcast_b") else L, case["N"])
    if op == "cdist":
        state["p"] = case["p"]
        state["skip_epilogue"] = bool(case.get("skip_epilogue", False))
        state["out"] = _out_buffer(case, L, case["M"], case["N"])
        return state
    state["descriptor"] = DESCRIPTORS[case["kernel"]]
    state["options"] = dict(bandwidth=case["bandwidth"])
    if op == "kernel":
        if case.get("tensor_bandwidth"):
            state["options"]["bandwidth"] = torch.full((L,), case["bandwidth"], device="cuda")
        if case["regularization"]:
            state["options"]["regularization"] = case["regularization"]
        state["out"] = _out_buffer(case, L, case["M"], case["N"])
    else:
        state["c"] = torch.randn(case["O"], case["M"], generator=gen, device="cuda")
    return state


def run(state):
    op = state["op"]
    if op == "cdist":
        return kermac.cdist(state["a"], state["b"], out=state["out"], p=state["p"], skip_epilogue=state["skip_epilogue"])
    if op == "kernel":
        return kermac.run_kernel(state["descriptor"], state["a"], state["b"], out=state["out"], **state["options"])
    if op == "grad":
        return kermac.cdist_grad(state["a"], state["b"], state["c"], state["d"], p=state["p"])
    return kermac.kernel_matvec(state["descriptor"], state["a"], state["b"], state["c"], **state["options"])


# ------------------------------------------------------------------------------------ work
def work(case):
    """Bytes: each input read once, each result written once.  Operations: the definition's own, with a
    subtract, a power (one operation, or three for a fractional order) and an add per term."""
    op, L, M, N, K = case["op"], case["L"], case["M"], case["N"], case["K"]
    power = 1 if case.get("p", 2.0) in (1.0, 2.0) else 3
    pairs = L * M * N
    if op == "grad":
        O = case["O"]
        return {"bytes": 4 * L * (K * M + N * K + O * K + N * M + O * N * M), "flops": pairs * K * (1 + power + 2 * O)}
    points = L * M * K
    if not case.get("same"):
        points += (1 if case.get("broadcast_b") else L) * N * K
    if op == "matvec":
        O = case["O"]
        return {"bytes": 4 * (points + O * M + N * O), "flops": pairs * (3 * K + 2 * O)}
    # K(X, X) is symmetric: half of its entries are enough
    terms = pairs // 2 if case.get("same") else pairs
    return {"bytes": 4 * (points + pairs), "flops": terms * K * (2 + power)}


def tolerance(case):
    """Everything is 32-bit: sums of K (or M) rounded terms, approximate square roots and exponentials."""
    return {"rel": 1e-5}
