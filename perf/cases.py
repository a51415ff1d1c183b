"""What is measured of the self-join engine: its public calls over the range of real use.

Every case is one pass of a program that has its points on the GPU (or, for the
estimator, its training batch) and an engine context in hand, and calls the
`sjoin` package: set the points, build the grid index, then join (pair count and
set hash of the device-resident result batches), list the pairs on the host,
fill the on-device CSR neighbour table, or count the neighbours of every point.
The estimator case is one loss and gradient of the scheduler's network.

Point sets are the generators of the repository's configurations and tests
(uniform, exponential with rate 40 clipped to [0, 1], a mixture of 64 Gaussians
with 10 % uniform background), drawn on the GPU from the seed.  Each listed case
stands for a family of calls; `draw` varies the family's size, radius, traversal
and precision over the range its comment states.

The order of the values inside one key's row is unspecified for the symmetric
traversals, so the calls that return pairs use the full stencil, whose rows come
in candidate order.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG_DIR = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "self-join-hpbdc2019_b200")
if _PKG_DIR not in sys.path:
    sys.path.insert(0, _PKG_DIR)

import sjoin  # noqa: E402

_WEIGHTS = os.path.join(sjoin.PKG, "estimator_c4.bin")
_RATE = 40.0


def _case(call, kind, n, dim, indexed, eps, mode, fp32=False, learned=False, capacity=0):
    return dict(call=call, kind=kind, n=int(n), dim=int(dim), indexed=int(indexed), eps=float(eps), mode=int(mode),
                fp32=bool(fp32), learned=bool(learned), capacity=int(capacity))


def listed():
    return [
        # a small set joined on demand: launches, host round trips and the task
        # builder are the time (2-D, 3,000 to 60,000 points)
        dict(_case("join", "exp", 20_000, 2, 2, 0.002, 10), name="join2d_20k"),
        # sorted pairs of a small 2-D set on the host in one batch (5,000 to 100,000 points, 8 to 31 neighbours)
        dict(_case("pairs", "uniform", 100_000, 2, 2, 0.01, 3), name="pairs2d_100k"),
        # the neighbour table in a device buffer that the program keeps (3-D, 10,000 to 250,000 points, 4 to 16 neighbours)
        dict(_case("csr", "uniform", 250_007, 3, 3, 0.02, 9), name="csr3d_250k"),
        # neighbour counts (density estimates) with fewer indexed dimensions than data dimensions
        dict(_case("degrees", "uniform", 200_003, 5, 3, 0.12, 4), name="degrees5d_200k"),
        # B-Unicomp in plain FP64, many batches of at most 5e7 pairs, skewed 2-D data
        dict(_case("join", "exp", 2_000_000, 2, 2, 0.0015, 5, capacity=50_000_000), name="join2d_2m"),
        # linear-ID Unicomp, FP32 filter with FP64 refinement, batches of 1e8 pairs, 4-D
        dict(_case("join", "exp", 1_500_000, 4, 4, 0.01, 6, fp32=True, capacity=100_000_000), name="join4d_1500k"),
        # the dense 6-D workload with the learned scheduler and batches of 2e9 pairs: the largest
        dict(_case("join", "exp", 1_500_000, 6, 6, 0.03, 10, fp32=True, learned=True, capacity=2_000_000_000),
             name="join6d_1500k"),
        # the same data in plain FP64 with the sampling scheduler
        dict(_case("join", "exp", 400_000, 6, 6, 0.03, 10, capacity=500_000_000), name="join6d_fp64_400k"),
        # clustered 16-D data indexed on six dimensions: many cells, few pairs
        dict(_case("join", "gauss", 1_000_000, 16, 6, 0.05, 10, fp32=True, learned=True), name="join16d_1m"),
        # full stencil over a work queue, padded width 8, fewer indexed dimensions
        dict(_case("join", "exp", 100_003, 8, 4, 0.05, 9, fp32=True), name="join8d_100k"),
        # neighbour counts of the dense 6-D data (the count pass alone)
        dict(_case("degrees", "exp", 600_011, 6, 6, 0.03, 10, fp32=True), name="degrees6d_600k"),
        # one training step's loss and gradient of the scheduler's network on the device
        dict(call="mlp_grad", n=8192, name="mlp_grad_8192"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.randrange(12)
    if family == 0:
        return _case("join", "exp", _log_int(rng, 3_000, 60_000), 2, 2, rng.uniform(0.001, 0.003),
                     rng.choice([3, 5, 6, 10]), fp32=rng.random() < 0.5)
    if family == 1:
        n = _log_int(rng, 5_000, 100_000)
        return _case("pairs", "uniform", n, 2, 2, math.sqrt(rng.uniform(8, 31) / (math.pi * n)), rng.choice([3, 9]),
                     fp32=rng.random() < 0.5)
    if family == 2:
        n = _log_int(rng, 10_000, 250_000)
        return _case("csr", "uniform", n, 3, 3, (rng.uniform(4, 16) / (4.0 / 3.0 * math.pi * n)) ** (1.0 / 3.0),
                     rng.choice([3, 9]), fp32=rng.random() < 0.5)
    if family == 3:
        return _case("degrees", "uniform", _log_int(rng, 20_000, 200_000), 5, 3, rng.uniform(0.08, 0.12),
                     rng.choice([3, 4, 6, 10]), fp32=rng.random() < 0.5)
    if family == 4:
        return _case("join", "exp", _log_int(rng, 200_000, 2_000_000), 2, 2, rng.uniform(0.0006, 0.0015),
                     rng.choice([4, 5, 6, 10]), capacity=50_000_000)
    if family == 5:
        return _case("join", "exp", _log_int(rng, 150_000, 1_500_000), rng.choice([3, 4]), 3, rng.uniform(0.005, 0.007),
                     rng.choice([6, 10]), fp32=True, capacity=100_000_000)
    if family == 6:
        return _case("join", "exp", _log_int(rng, 150_000, 1_500_000), 6, 6, rng.uniform(0.015, 0.03), 10, fp32=True,
                     learned=rng.random() < 0.5, capacity=2_000_000_000)
    if family == 7:
        return _case("join", "exp", _log_int(rng, 50_000, 400_000), rng.choice([5, 6]), 5, rng.uniform(0.015, 0.025),
                     rng.choice([4, 6, 10]), capacity=500_000_000)
    if family == 8:
        return _case("join", "gauss", _log_int(rng, 100_000, 1_000_000), 16, 6, rng.uniform(0.03, 0.05), 10, fp32=True,
                     learned=rng.random() < 0.5)
    if family == 9:
        return _case("join", "exp", _log_int(rng, 10_000, 100_000), rng.choice([7, 8, 12]), 4, rng.uniform(0.03, 0.05),
                     rng.choice([3, 7, 8, 9]), fp32=rng.random() < 0.5)
    if family == 10:
        return _case("degrees", "exp", _log_int(rng, 60_000, 600_000), 6, 6, rng.uniform(0.015, 0.03),
                     rng.choice([6, 10]), fp32=True)
    return dict(call="mlp_grad", n=_log_int(rng, 1, 8192))


def _points(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    n, d = case["n"], case["dim"]

    def uniform(*shape):
        return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)

    if case["kind"] == "uniform":
        return uniform(n, d)
    if case["kind"] == "exp":
        return torch.clamp(-torch.log1p(-uniform(n, d)) / _RATE, 0.0, 1.0)
    background = int(round(0.10 * n))
    centre, sigma = uniform(64, d), 0.02 + 0.06 * uniform(64)
    which = torch.randint(0, 64, (n - background,), generator=g, device="cuda")
    noise = torch.randn((n - background, d), generator=g, device="cuda", dtype=torch.float64)
    pts = torch.cat([centre[which] + noise * sigma[which][:, None], uniform(background, d)])
    return pts[torch.randperm(n, generator=g, device="cuda")].contiguous()


def _batch(case, seed):
    """Standardised features and two targets, as the estimator's training sees them."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 29)
    x = torch.randn((case["n"], 16), generator=g, device="cuda")
    y = torch.stack([x[:, :4].sum(1), x[:, 4:8].abs().sum(1)], 1).contiguous()
    return x, y, torch.from_numpy(sjoin.mlp_init(int(seed) % 1000)).cuda()


def prepare(case, seed):
    if case["call"] == "mlp_grad":
        x, y, w = _batch(case, seed)
        return dict(case=case, x=x, y=y, w=w, loss=torch.zeros(1, device="cuda"), grad=torch.zeros_like(w))
    sj = sjoin.SelfJoin(case["dim"], case["eps"], indexed_dims=case["indexed"], mode=case["mode"],
                        precision=sjoin.PREC_FP32_REFINE if case["fp32"] else sjoin.PREC_FP64,
                        scheduler=sjoin.SCHED_LEARNED if case["learned"] else sjoin.SCHED_SAMPLING,
                        capacity=case["capacity"])
    if case["learned"]:
        sj.load_estimator(_WEIGHTS)
    state = dict(case=case, sj=sj, pts=_points(case, seed))
    # result buffers that such a program keeps, with room above the expected pairs (unused slots -1)
    if case["call"] == "pairs":
        state.update(keys=np.full(_room(case), -1, np.int32), vals=np.full(_room(case), -1, np.int32))
    elif case["call"] == "csr":
        state.update(row=torch.zeros(case["n"] + 1, dtype=torch.int64, device="cuda"),
                     cols=torch.full((_room(case),), -1, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()   # the engine reads the points on its own stream
    return state


def run(state):
    case = state["case"]
    if case["call"] == "mlp_grad":
        sjoin.mlp_loss_grad_noalloc(state["x"].data_ptr(), state["y"].data_ptr(), case["n"], state["w"].data_ptr(),
                                    state["loss"].data_ptr(), state["grad"].data_ptr(),
                                    torch.cuda.current_stream().cuda_stream)
        return dict(loss=state["loss"], grad=state["grad"])
    sj, pts = state["sj"], state["pts"]
    sj.set_points_device(pts.data_ptr(), case["n"])
    sj.build_index()
    if case["call"] == "join":
        st = sj.join(sjoin.DELIVER_NONE)
        return dict(pairs=int(st.total_pairs), hash=np.array([st.pair_hash], dtype=np.uint64).view(np.int64))
    if case["call"] == "pairs":
        keys, vals, at = state["keys"], state["vals"], [0]

        def take(_batch, key, val):
            keys[at[0]:at[0] + len(key)] = key
            vals[at[0]:at[0] + len(val)] = val
            at[0] += len(key)

        sj.join(sjoin.DELIVER_HOST, take)
        return dict(pairs=at[0], keys=keys, vals=vals)
    if case["call"] == "degrees":
        return dict(degrees=sj.degrees().view(np.int32))
    total = sj.neighbor_csr(state["row"].data_ptr(), state["cols"].data_ptr(), state["cols"].numel())
    return dict(pairs=total, row=state["row"], cols=state["cols"])


def _expected_pairs(case):
    """Expected result pairs, self pairs included: the radius ball's volume for
    uniform points (the border neglected), a fixed Monte Carlo sample of point
    pairs for exponential ones; the Gaussian mixture has few beyond the self pairs."""
    n, d, eps = case["n"], case["dim"], case["eps"]
    if case["kind"] == "uniform":
        return n + n * float(n) * math.pi ** (d / 2) / math.gamma(d / 2 + 1) * eps ** d
    if case["kind"] == "gauss":
        return 1.1 * n
    r = np.random.default_rng(1)
    a, b = (np.clip(-np.log1p(-r.random((2048, d))) / _RATE, 0.0, 1.0) for _ in range(2))
    d2 = sum((a[:, None, j] - b[None, :, j]) ** 2 for j in range(d))
    return n + n * float(n) * float(np.mean(d2 <= eps * eps))


def _room(case):
    return int(1.05 * _expected_pairs(case)) + 10_000


def work(case):
    n = case["n"]
    if case["call"] == "mlp_grad":
        weights = 16 * 64 + 64 * 64 + 64 * 2
        return dict(bytes=4 * (18 * n + 2 * 5378 + 1), flops=2 * n * (3 * weights - 16 * 64))
    pairs = _expected_pairs(case)
    out = {"join": 8 * pairs, "pairs": 8 * pairs, "degrees": 4 * n, "csr": 4 * pairs + 8 * (n + 1)}[case["call"]]
    # every unordered result pair's squared distance has to be evaluated once
    return dict(bytes=8 * n * case["dim"] + out, flops=3 * case["dim"] * pairs / 2)


def _exact_degrees(case, seed):
    n, d = case["n"], case["dim"]
    if float(n) * n * d > 2.5e11:
        return None
    p = _points(case, seed)
    deg = torch.zeros(n, dtype=torch.int64, device="cuda")
    step = max(1, int(2e8 // n))
    for i in range(0, n, step):
        acc = torch.zeros((min(step, n - i), n), dtype=torch.float64, device="cuda")
        for j in range(d):
            acc += (p[i:i + step, j, None] - p[None, :, j]) ** 2
        deg[i:i + step] = (acc.sqrt() <= case["eps"]).sum(1)
    return deg


def exact(case, seed):
    if case["call"] == "mlp_grad":
        x, y, w = (t.double() for t in _batch(case, seed))
        w.requires_grad_(True)
        w1, b1, w2, b2, w3, b3 = torch.split(w, [1024, 64, 4096, 64, 128, 2])
        h = torch.relu(x @ w1.view(16, 64) + b1)
        h = torch.relu(h @ w2.view(64, 64) + b2)
        loss = 0.5 * ((h @ w3.view(64, 2) + b3 - y) ** 2).sum() / case["n"]
        loss.backward()
        return dict(loss=loss.detach().view(1), grad=w.grad)
    deg = _exact_degrees(case, seed)
    if deg is None:
        return None
    if case["call"] == "join":
        return dict(pairs=int(deg.sum()), hash=None)
    if case["call"] == "pairs":
        keys = np.full(_room(case), -1, np.int32)
        listed_keys = torch.repeat_interleave(torch.arange(case["n"], device="cuda"), deg).int().cpu().numpy()
        keys[:len(listed_keys)] = listed_keys
        return dict(pairs=len(listed_keys), keys=keys, vals=None)
    if case["call"] == "degrees":
        return dict(degrees=deg.int().cpu().numpy())
    row = torch.zeros(case["n"] + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.cumsum(deg, 0)
    return dict(pairs=int(row[-1]), row=row, cols=None)
