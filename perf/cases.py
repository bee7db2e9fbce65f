"""The work a user of this package has it do, as timed cases.

Three ways in are covered: the scikit-learn-style estimator on host arrays (``KMeans``), the resident handle on a
matrix that already lives on the GPU (``ResidentKMeans``), and the predict / transform of a fitted model on new host data
(``KMeansH2O``).
Sizes come from the benchmark configurations (100,000 x 32 ... 10,000,000 x 64, 128 / 256 / 784 columns, 8 ... 4096
centroids, float32 and float64), the test fixtures (2,000 x 32) and the colour-quantisation picture of the baseline
table (273,280 x 3 float64, 64 colours), or are generic.

A case is a dict: ``kind`` (which calls are made), ``n`` rows, ``d`` columns, ``k`` centroids, ``iters`` (Lloyd
iterations, or their limit for the estimator), ``dtype`` of the matrix, ``data`` (how it is distributed), and, for the
estimator's fit, ``weights`` (sample weights) and ``tol``.
"""
import numpy as np
import torch

from h2o4gpu_b200 import KMeans, KMeansH2O, ResidentKMeans

# value distributions, as in the benchmark configurations: centre half-range or spread and noise of the mixtures
MIXTURES = {
    "blobs": dict(half=10.0, sigma=1.0, dirichlet=False),     # equal-weight mixture
    "uneven": dict(half=10.0, sigma=1.0, dirichlet=True),     # Dirichlet(1) mixing weights
    "spread": dict(half=20.0, sigma=2.0, dirichlet=False),    # wider centres, sigma 2
    "offset": dict(half=3.5, sigma=1.0, dirichlet=False),     # standard normal plus an offset of variance 4
}
NP_DTYPES = {"float32": np.float32, "float64": np.float64, "uint8": np.uint8}


def listed():
    return [
        # a small host array through the estimator with its defaults (k-means|| start, tolerance test): pure latency
        dict(name="fit_small_array", kind="estimator_fit", n=2_000, d=32, k=8, iters=300, dtype="float32",
             data="blobs", weights=False, tol=1e-4),
        # colour quantisation of one picture: three float64 columns, 64 colours, fit until it converges
        dict(name="fit_colours", kind="estimator_fit", n=273_280, d=3, k=64, iters=300, dtype="float64",
             data="colours", weights=False, tol=1e-4),
        # 8-bit pixels with sample weights through the estimator: typed upload, weighted sums
        dict(name="fit_pixels_weighted", kind="estimator_fit", n=200_000, d=784, k=10, iters=10, dtype="uint8",
             data="images", weights=True, tol=0.0),
        # few centroids, narrow rows, fits in L2: launches count
        dict(name="fit_k8_d32", kind="fit", n=100_000, d=32, k=8, iters=20, dtype="float32", data="blobs"),
        # the benchmark's headline shape: bound by the memory
        dict(name="fit_k100_d64", kind="fit", n=10_000_000, d=64, k=100, iters=20, dtype="float32", data="uneven"),
        # many centroids: the tensor cores' share grows
        dict(name="fit_k1000_d128", kind="fit", n=2_000_000, d=128, k=1000, iters=10, dtype="float32", data="spread"),
        # image-like rows (mostly zero), few centroids, wide rows
        dict(name="fit_k10_d784", kind="fit", n=500_000, d=784, k=10, iters=20, dtype="float32", data="images"),
        # the contraction-bound shape
        dict(name="fit_k4096_d256", kind="fit", n=500_000, d=256, k=4096, iters=10, dtype="float32", data="offset"),
        # the same in float64
        dict(name="fit_k4096_d256_f64", kind="fit", n=60_000, d=256, k=4096, iters=5, dtype="float64", data="offset"),
        # labels of a resident matrix of odd sizes (rows not 16-byte aligned)
        dict(name="assign_k37_d50", kind="assign", n=1_000_003, d=50, k=37, iters=0, dtype="float32", data="blobs"),
        # labels of a new host array
        dict(name="predict_array", kind="predict", n=1_000_000, d=64, k=100, iters=0, dtype="float32", data="uneven"),
        # all distances of a new host array
        dict(name="transform_array", kind="transform", n=300_000, d=784, k=100, iters=0, dtype="float32", data="images"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case: kinds as a user mixes them, sizes spread over their logarithm, odd ones among them."""
    kind = rng.choice(["fit", "fit", "fit", "fit", "estimator_fit", "assign", "predict", "transform"])
    dtype = "float64" if rng.random() < 0.2 else "float32"
    d = _log(rng, 2, 1024)
    if rng.random() < 0.5:
        d = max(2, d // 8 * 8)
    if kind == "fit":
        n, k = _log(rng, 5_000, 10_000_000), _log(rng, 2, 4096)
        iters = rng.choice([5, 10, 20])
    elif kind == "estimator_fit":
        n, k = _log(rng, 1_000, 500_000), _log(rng, 2, 128)
        iters = rng.choice([20, 50, 300])
    else:
        n, k = _log(rng, 1_000, 4_000_000), _log(rng, 2, 1000)
        iters = 0
    size = 8 if dtype == "float64" else 4
    n = min(n, int((1 << 31) // (d * size)) if kind in ("fit", "assign") else int((1 << 28) // (d * size)))
    if kind == "transform":
        n = min(n, int((1 << 27) // (k * size)))
    # the arithmetic of a case stays below that of the largest listed ones
    most = 1e11 if dtype == "float64" else 1e12
    n = max(1_000, min(n, int(most / (float(k) * d * (max(iters, 1) + 1)))))
    k = min(k, max(2, n // 8))
    data = "images" if d >= 256 and k <= 128 and rng.random() < 0.5 else rng.choice(["blobs", "uneven", "spread", "offset"])
    case = dict(kind=kind, n=n, d=d, k=k, iters=iters, dtype=dtype, data=data)
    if kind == "estimator_fit":
        case["weights"] = rng.random() < 0.25
        case["tol"] = 0.0 if case["weights"] else rng.choice([0.0, 1e-4])
        if data == "images" and rng.random() < 0.5:
            case["dtype"] = "uint8"
    return case


def _matrix(case, g):
    """n x d on the GPU in the case's dtype, and the generating centres (or None)."""
    n, d, k = case["n"], case["d"], case["k"]
    out = {"float32": torch.float32, "float64": torch.float64, "uint8": torch.uint8}[case["dtype"]]
    work = torch.float64 if out == torch.float64 else torch.float32
    X = torch.empty((n, d), dtype=out, device="cuda")
    step = max(1, (1 << 26) // d)
    if case["data"] == "images":      # 0 with probability 0.8, else an integer in 1..255
        for s in range(0, n, step):
            m = min(step, n - s)
            v = torch.randint(1, 256, (m, d), generator=g, device="cuda", dtype=torch.int32)
            v[torch.rand((m, d), generator=g, device="cuda") < 0.8] = 0
            X[s:s + m] = v.to(out)
        return X, None
    if case["data"] == "colours":     # smooth gradients with noise, scaled to [0, 1] as picture libraries return them
        comp = torch.rand((256, d), generator=g, device="cuda", dtype=work)
        which = torch.randint(0, 256, (n,), generator=g, device="cuda")
        t = torch.rand((n, 1), generator=g, device="cuda", dtype=work)
        v = comp[which] * t + comp[(which + 1) % 256] * (1 - t)
        v = v + 0.02 * torch.randn((n, d), generator=g, device="cuda", dtype=work)
        X[:] = (torch.round(v.clamp(0, 1) * 255) / 255).to(out)
        return X, None
    p = MIXTURES[case["data"]]
    half = max(p["half"], 3.0 * p["sigma"] * k ** (1.0 / d))      # in few columns the components stay apart too
    centers = (torch.rand((k, d), generator=g, device="cuda", dtype=work) * 2 - 1) * half
    if p["dirichlet"]:
        w = -torch.log(torch.rand((k,), generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-300))
        edges = torch.cumsum(w / w.sum(), 0)
    for s in range(0, n, step):
        m = min(step, n - s)
        if p["dirichlet"]:
            u = torch.rand((m,), generator=g, device="cuda", dtype=torch.float64)
            which = torch.searchsorted(edges, u).clamp_max(k - 1)
        else:
            which = torch.randint(0, k, (m,), generator=g, device="cuda")
        X[s:s + m] = centers[which] + p["sigma"] * torch.randn((m, d), generator=g, device="cuda", dtype=work)
    return X, centers


class _DeviceLabels(object):
    """The handle's label buffer as an array on the GPU; keeps the handle alive."""

    def __init__(self, handle, rows):
        self.handle = handle
        self.__cuda_array_interface__ = {"shape": (rows,), "typestr": "<i4", "version": 3, "strides": None,
                                         "data": (handle.labels_device_ptr(0), False)}


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1_000_003 + 17)
    X, centers = _matrix(case, g)
    n, d, k = case["n"], case["d"], case["k"]
    state = {"case": case}
    kind = case["kind"]
    dtype = NP_DTYPES["float64" if case["dtype"] == "float64" else "float32"]
    rows = torch.randperm(n, generator=g, device="cuda")[:k]
    if kind in ("fit", "assign"):
        # initial centroids: seeded random rows; labels are asked for with centroids as a fit leaves them
        init = X[rows] if kind == "fit" or centers is None else centers
        state["X"] = X
        state["init"] = init.cpu().numpy().astype(dtype)
        state["handle"] = ResidentKMeans(dtype=dtype, devices=(0,))
    elif kind == "estimator_fit":
        state["X"] = X.cpu().numpy()
        state["w"] = (torch.rand((n,), generator=g, device="cuda") + 0.5).cpu().numpy() if case["weights"] else None
        state["seed"] = int(seed) % 32000
    else:
        host = X.cpu().numpy()
        # a model as it was fitted earlier and is loaded again: its centres are known
        model = KMeansH2O(n_clusters=k)
        model.cluster_centers_ = (X[rows] if centers is None else centers).cpu().numpy().astype(dtype)
        state["X"], state["model"] = host, model
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fit":
        h, X = state["handle"], state["X"]
        h.attach_device(0, X.data_ptr(), case["n"], case["d"])
        h.fit(state["init"], case["iters"])
        return {"centers": h.centroids(), "labels": torch.as_tensor(_DeviceLabels(h, case["n"]), device="cuda")}
    if kind == "assign":
        h, X = state["handle"], state["X"]
        h.attach_device(0, X.data_ptr(), case["n"], case["d"])
        h.set_centroids(state["init"])
        h.assign()
        return {"labels": torch.as_tensor(_DeviceLabels(h, case["n"]), device="cuda")}
    if kind == "estimator_fit":
        m = KMeans(n_clusters=case["k"], max_iter=case["iters"], tol=case["tol"], random_state=state["seed"])
        m.fit(state["X"], sample_weight=state["w"])
        return {"centers": m.cluster_centers_, "labels": m.labels_, "inertia": float(m.inertia_)}
    if kind == "predict":
        return {"labels": state["model"].predict(state["X"])}
    return {"distances": state["model"].transform(state["X"])}


def work(case):
    n, d, k, it = case["n"], case["d"], case["k"], case["iters"]
    size = {"float32": 4, "float64": 8, "uint8": 1}[case["dtype"]]
    rows, table = float(n) * d * size, float(k) * d * size
    kind = case["kind"]
    if kind == "fit":
        # every assignment reads the rows once (the sums of an update can share that reading) and leaves one label
        # per row; the closing assignment makes one pass more
        return {"bytes": (it + 1) * (rows + 4.0 * n) + 2 * table, "flops": (it + 1) * 2.0 * n * d * k}
    if kind == "estimator_fit":
        # how many iterations it takes until it converges depends on the data: one reading is what is sure
        return {"bytes": rows + 4.0 * n + table, "flops": 2.0 * n * d * k}
    if kind == "transform":
        return {"bytes": rows + float(n) * k * size + table, "flops": 2.0 * n * d * k}
    return {"bytes": rows + 4.0 * n + table, "flops": 2.0 * n * d * k}


def tolerance(case):
    # Measured by running each kind in float32 and in float64 on the same values.  In one assignment up to 2.5e-5 of
    # the rows were equally far from two centroids to rounding (two columns, 395 clusters; none on most shapes);
    # distances differed by 1e-7, more where |x|^2 + |c|^2 - 2 x.c cancels.  A fit repeats assignments on its own
    # results, so such rows can move others after them: 9e-5 of the centres and 9e-4 of the labels on overlapping
    # clusters, and, on images of pure noise (no clusters at all), 5e-3 and 1e-2.
    kind, f64 = case["kind"], case["dtype"] == "float64"
    few = 2.0 / case["n"]                                          # two rows of a small matrix
    if kind in ("assign", "predict"):
        return {"rel": 0.0, "differ": max(few, 1e-6 if f64 else 1e-4)}
    if kind == "transform":
        return {"rel": 1e-12 if f64 else 1e-5}
    if f64:
        return {"rel": 1e-9, "differ": 1e-6}
    if case["data"] == "images":
        return {"rel": 2e-2, "max": 0.99, "differ": 1e-2}
    return {"rel": 4e-4, "max": 8e-3, "differ": max(few, 4e-3)}
