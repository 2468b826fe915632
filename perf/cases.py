"""Performance cases of the engine: what a program that uses it has it do.

Three kinds of pass, each through the public interface:

  matvec  y = K q on an assembled AFMM (the setup is done once, many products follow), with device or host
          vectors, in every precision, for one and for several right-hand sides;
  set     one product of many small problems in one call (AFMMSet);
  setup   the whole of a one-shot program: construct, assemble, one product (and read back the permutation and
          the ranks), the sequence of the reference's example programs.

Sizes, kernels and tolerances are those of the package's workloads and benchmark, with odd and ragged sizes
among them.  Charges are standard normal; points are uniform, a 16-component Gaussian mixture, or a spiral in a
uniform background.
"""
import math

import numpy as np
import torch

from afmm2d_b200 import AFMM, AFMMSet

GAUSS_PARAM = 0.01


def listed():
    return [
        # the smallest product a program repeats: launch latency and the depth of the tree count
        dict(name="fp64_4k_log", kind="matvec", N=4096, kernel="log", points="uniform", M=32, tol=8,
             precision="fp64", nrhs=1, where="device", storage="auto"),
        # the ordinary single product at the reference's published size, a tight tolerance
        dict(name="fp64_1m_log", kind="matvec", N=1048576, kernel="log", points="uniform", M=64, tol=10,
             precision="fp64", nrhs=1, where="device", storage="auto"),
        # the reference's own call: host vector in, host vector out, an odd size, the example program's kernel
        dict(name="fp64_100k_scaled_host", kind="matvec", N=100003, kernel="one_over_r_scaled", points="uniform",
             M=100, tol=6, precision="fp64", nrhs=1, where="host", storage="auto"),
        # one right-hand side in mixed precision on clustered points, a ragged tree
        dict(name="mixed_300k_mixture", kind="matvec", N=300000, kernel="one_over_r", points="mixture", M=64, tol=6,
             precision="mixed", nrhs=1, where="device", storage="auto"),
        # the largest: 16 right-hand sides, mixed precision, 4M clustered points (the package's headline workload)
        dict(name="mixed16_4m_mixture", kind="matvec", N=4194304, kernel="one_over_r", points="mixture", M=64, tol=6,
             precision="mixed", nrhs=16, where="device", storage="auto"),
        # many right-hand sides in FP64 throughout (a block solver that needs full accuracy)
        dict(name="fp64b16_1m_log", kind="matvec", N=1048576, kernel="log", points="uniform", M=64, tol=10,
             precision="fp64_batched", nrhs=16, where="device", storage="auto"),
        # many right-hand sides of a smooth kernel
        dict(name="mixed64_1m_gauss", kind="matvec", N=1048576, kernel="gaussian", points="uniform", M=64, tol=8,
             precision="mixed", nrhs=64, where="device", storage="auto"),
        # a few right-hand sides (an unfilled pass) at an odd size
        dict(name="fp64b5_100k_log", kind="matvec", N=100003, kernel="log", points="uniform", M=32, tol=8,
             precision="fp64_batched", nrhs=5, where="device", storage="auto"),
        # blocks that are not stored (the policy of problems too large for the memory): entries on the fly
        dict(name="fp64_otf_256k_spiral", kind="matvec", N=262144, kernel="log", points="spiral", M=64, tol=12,
             precision="fp64", nrhs=1, where="device", storage="on_the_fly"),
        # many small problems in one call
        dict(name="set48_2k_64k_log", kind="set", count=48, nmin=2048, nmax=65536, kernel="log", points="uniform",
             M=32, tol=8),
        # a one-shot program at a middling size, tight tolerance
        dict(name="setup_256k_log", kind="setup", N=262144, kernel="log", points="uniform", M=64, tol=10),
        # a one-shot program on clustered points
        dict(name="setup_500k_mixture", kind="setup", N=500000, kernel="one_over_r", points="mixture", M=64, tol=6),
    ]


# kernel, points, leaf sizes, tolerances, largest N: the combinations that the workloads use
FAMILIES = [
    ("log", "uniform", (32, 64), (6, 8, 10), 2 << 20),
    ("one_over_r", "mixture", (64,), (4, 6), 4 << 20),
    ("gaussian", "uniform", (64,), (6, 8), 2 << 20),
    ("one_over_r_scaled", "uniform", (64, 100), (4, 6, 8), 1 << 20),
    ("log", "spiral", (64,), (8, 12), 1 << 18),
]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kernel, points, leaf, tols, nmax = rng.choice(FAMILIES)
    base = dict(kernel=kernel, points=points, M=rng.choice(leaf), tol=rng.choice(tols))
    kind = rng.choice(["matvec"] * 7 + ["set", "setup"])
    if kind == "set":
        base.update(kernel="log", points="uniform", M=32, tol=rng.choice((6, 8)))
        lo = _log_size(rng, 2048, 16384)
        return dict(kind="set", count=_log_size(rng, 4, 48), nmin=lo, nmax=_log_size(rng, lo, 65536), **base)
    if kind == "setup":
        return dict(kind="setup", N=_log_size(rng, 4096, min(nmax, 1 << 20) // (2 if points == "spiral" else 1)), **base)
    precision = rng.choice(["fp64", "fp64", "mixed", "mixed", "fp64_batched"])
    N = _log_size(rng, 16 * base["M"] + 1, nmax)
    if precision == "fp64":
        nrhs = rng.choice([1, 1, 1, 2])
    elif precision == "mixed":
        nrhs = rng.choice([1, 1, _log_size(rng, 2, 16), 16, 32])
    else:
        nrhs = rng.choice([_log_size(rng, 2, 16), 16])
    while N * nrhs > 1 << 26:
        nrhs //= 2
    where = "host" if rng.random() < 0.2 and N * nrhs <= 1 << 21 else "device"
    storage = "on_the_fly" if precision == "fp64" and rng.random() < 0.15 and N <= 1 << 19 else "auto"
    return dict(kind="matvec", N=N, precision=precision, nrhs=nrhs, where=where, storage=storage, **base)


def _points(kind, N, rng):
    if kind == "uniform":
        return rng.uniform(0.0, 1.0, size=(N, 2))
    if kind == "mixture":
        centres = rng.uniform(0.0, 1.0, size=(16, 2))
        return centres[rng.integers(0, 16, size=N)] + 0.02 * rng.standard_normal((N, 2))
    h = N // 2
    theta = rng.uniform(0.0, 20 * np.pi, size=h)
    arm = 0.05 * theta[:, None] * np.stack([np.cos(theta), np.sin(theta)], axis=1)
    arm += 1e-4 * rng.standard_normal((h, 2))
    return np.concatenate([arm, rng.uniform(arm.min(axis=0), arm.max(axis=0), size=(N - h, 2))])


def _sizes(case):
    """The sizes of a set's problems: log-uniform, the same for every seed."""
    rng = np.random.Generator(np.random.PCG64(case["count"]))
    return [int(round(math.exp(x))) for x in
            rng.uniform(math.log(case["nmin"]), math.log(case["nmax"] + 1e-9), size=case["count"])]


def _inputs(case, seed):
    """(points, charges): host arrays, charges (nrhs, N) or (N,); for a set, lists of them."""
    rng = np.random.Generator(np.random.PCG64(seed))
    if case["kind"] == "set":
        pts = [_points(case["points"], n, rng) for n in _sizes(case)]
        return pts, [rng.standard_normal(len(p)) for p in pts]
    pts = _points(case["points"], case["N"], rng)
    nrhs = case.get("nrhs", 1)
    if case["N"] * nrhs <= 1 << 21:
        return pts, rng.standard_normal((nrhs, case["N"]))
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1)
    return pts, torch.randn((nrhs, case["N"]), dtype=torch.float64, device="cuda", generator=g)


def _afmm(case, pts):
    kparam = GAUSS_PARAM if case["kernel"] == "gaussian" else None
    return AFMM(len(pts), case["M"], case["tol"], pts, kernel=case["kernel"], kparam=kparam)


def prepare(case, seed):
    pts, q = _inputs(case, seed)
    if case["kind"] == "setup":
        return dict(case=case, pts=pts, q=q[0] if isinstance(q, np.ndarray) else q[0].cpu().numpy())
    if case["kind"] == "set":
        problems = []
        for p in pts:
            a = _afmm(case, p)
            a.assemble()
            problems.append(a)
        qd = torch.from_numpy(np.concatenate(q)).cuda()
        return dict(case=case, afmm=AFMMSet(problems), q=qd, y=torch.empty_like(qd))
    a = _afmm(case, pts)
    if case["storage"] != "auto":
        a.set_m2l_storage(case["storage"])
    a.assemble()
    if case["where"] == "host":
        q = q if isinstance(q, np.ndarray) else q.cpu().numpy()
        return dict(case=case, afmm=a, q=q[0] if case["nrhs"] == 1 else np.ascontiguousarray(q.T))
    qd = torch.from_numpy(q).cuda() if isinstance(q, np.ndarray) else q
    return dict(case=case, afmm=a, q=qd, y=torch.empty_like(qd))


def run(state):
    case = state["case"]
    if case["kind"] == "setup":
        a = _afmm(case, state["pts"])
        a.assemble()
        y = a.computeMatVecProduct(state["q"])
        levels = range(2, a.nLevels + 1)
        out = dict(y=y, permutation=a.permutation(), ranks=[a.ranks(j) for j in levels])
        a.close()
        return out
    a = state["afmm"]
    if case["kind"] == "set":
        a.matvec_device(state["q"].data_ptr(), state["y"].data_ptr())
        return state["y"]
    if case["where"] == "host":
        return a.computeMatVecProduct(state["q"], case["precision"])
    a.matvec_device(state["q"].data_ptr(), state["y"].data_ptr(), case["nrhs"], case["N"], case["precision"])
    return state["y"]


def _levels(N, M):
    return int(math.log(N // M) / math.log(4.0))


# typical skeleton size of a box, by kernel and tolerance: it sizes the operators that a product has to apply
def _rank(case):
    per_digit = {"log": 3.1, "one_over_r": 5.5, "one_over_r_scaled": 4.2, "gaussian": 1.9}[case["kernel"]]
    return per_digit * case["tol"] * (1.2 if case["points"] == "spiral" else 1.0)


def _product(case, N, nrhs):
    """Operations and bytes of one product: near-field entries once per unordered pair, the interpolation
    operators and the far-field blocks (also once per unordered pair of boxes), charges and potentials."""
    L = _levels(N, case["M"])
    leaves = 4 ** L
    per = N / leaves
    r = min(_rank(case), per)
    boxes = sum(4 ** j for j in range(2, L + 1))
    near = 0.5 * 9 * N * per
    far = 0.5 * 27 * boxes * r * r
    interp = leaves * per * r + (boxes - leaves) * 4 * r * r
    flops = near * (12 + 4 * nrhs) + far * 4 * nrhs + interp * 4 * nrhs
    entry = 4 if case.get("precision") == "mixed" else 8
    stored = 0 if case.get("storage") == "on_the_fly" else far * entry
    nbytes = stored + interp * 8 + 16 * N + 16 * N * nrhs
    if not stored:
        flops += far * 12
    return flops, nbytes


def work(case):
    if case["kind"] == "set":
        each = [_product(case, n, 1) for n in _sizes(case)]
        return dict(flops=sum(f for f, _ in each), bytes=sum(b for _, b in each))
    flops, nbytes = _product(case, case["N"], case.get("nrhs", 1))
    if case["kind"] == "setup":
        # cross approximation: r steps over the box's rows and its interaction list's columns, each step
        # against all earlier ones (residual and stopping test)
        L = _levels(case["N"], case["M"])
        per = case["N"] / 4 ** L
        r = min(_rank(case), per)
        boxes = sum(4 ** j for j in range(2, L + 1))
        flops += boxes * 28 * per * r * r * 2
        nbytes += 16 * case["N"]
    return dict(flops=flops, bytes=nbytes)


def _dense(case, pts, q):
    """K q in 64 bits, row block by row block; q (nrhs, N) -> (nrhs, N)."""
    x = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
    N = len(x)
    q = (torch.from_numpy(q) if isinstance(q, np.ndarray) else q).cuda()
    a = 0.5 ** _levels(N, case["M"])
    out = torch.empty((q.shape[0], N), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // N)
    for i in range(0, N, step):
        R2 = (x[i:i + step, None, 0] - x[None, :, 0]).square_()
        R2 += (x[i:i + step, None, 1] - x[None, :, 1]).square_()
        if case["kernel"] == "gaussian":
            K = R2.mul_(-1.0 / GAUSS_PARAM).exp_()
        elif case["kernel"] == "one_over_r":
            K = torch.where(R2 == 0, 0.0, R2.rsqrt())
        elif case["kernel"] == "one_over_r_scaled":
            R = R2.sqrt_()
            K = torch.where(R < a, R / a, a / R)
        else:
            K = torch.where(R2 < a * a, 0.5 / (a * a) * R2, 0.5) * R2.log()
            K = torch.where(R2 < 1e-10, 0.0, K)
        out[:, i:i + step] = q @ K.T
    return out


def exact(case, seed):
    if case["kind"] == "set":
        pts, q = _inputs(case, seed)
        return torch.cat([_dense(case, p, c[None])[0] for p, c in zip(pts, q)])
    # above this a dense product takes too long; on the clustered mixture the method itself is far from the
    # dense product (0.1 to 1 relative: its interaction lists take near boxes of the KD tree for far ones)
    if case["N"] > 600000 or case["points"] == "mixture":
        return None
    pts, q = _inputs(case, seed)
    y = _dense(case, pts, q)
    if case["kind"] == "setup":
        L = _levels(case["N"], case["M"])
        return dict(y=y[0], permutation=None, ranks=[None] * (L - 1))
    if case["where"] == "host":
        return y[0] if case["nrhs"] == 1 else y.T
    return y
