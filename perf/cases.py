"""The work whose speed is watched: what programs that use this library have it do.

listed() gives twelve cases and draw() more of the same ranges; prepare() makes what
a program holds before the call (device matrices, a plan, pinned host arrays), run()
is one pass through the public entry points, exact() the same result from torch in
64 bits.  Five kinds of work:

  posv     ppotrf / ppotrs / pposv / diag_logdet on a device matrix, all four types,
           both triangles; the matrix is copied into place first (the factor
           overwrites it), on the handle's stream, as a program that keeps A does
  mixed    pposv_mixed: FP64 accuracy from a TF32 / BF16 tensor-core factor
  host     pposv_mixed_host: the same from pinned host arrays
  batched  a VbatchedPlan replay: thousands of uneven matrices factored, solved and
           log-det'd in one launch
  gp       gp_nll and its gradient with respect to theta (one step of a GP fit)

Sizes and distributions are those of the benchmark configurations and the tests.
"""
import math

import numpy as np
import torch

from libddla_b200 import ddla
from libddla_b200.ddla import autograd, batched
from libddla_b200.workloads import householder_spd, se_kernel

TORCH = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
NUMPY = {"s": np.float32, "d": np.float64, "c": np.complex64, "z": np.complex128}
BYTES = {"s": 4, "d": 8, "c": 8, "z": 16}
DEV = "cuda"
_tuned = set()


def listed():
    return [
        # one small system: latency, launches and the host path are all of it
        dict(name="pposv_d_200", kind="posv", type="d", uplo="L", n=200, nrhs=1, pad=0, matrix="gram", split=False),
        # the plain configuration: factor, solve and log-determinant as three calls
        dict(name="potrf_potrs_logdet_d_2048", kind="posv", type="d", uplo="L", n=2048, nrhs=16, pad=0, matrix="gram",
             split=True),
        # an order (and so a leading dimension) that is odd, a ragged last block
        dict(name="pposv_d_5003", kind="posv", type="d", uplo="L", n=5003, nrhs=3, pad=0, matrix="gram", split=False),
        # the double and the complex kernel-matrix solves with many right-hand sides
        dict(name="pposv_d_16384", kind="posv", type="d", uplo="L", n=16384, nrhs=64, pad=0, matrix="se", split=False),
        dict(name="pposv_z_8192", kind="posv", type="z", uplo="L", n=8192, nrhs=64, pad=0, matrix="se", split=False),
        # single precision, upper triangle, padded leading dimension
        dict(name="pposv_s_upper_6000", kind="posv", type="s", uplo="U", n=6000, nrhs=32, pad=16, matrix="gram",
             split=False),
        # the headline solve: double accuracy from a low-precision factor
        dict(name="mixed_32768", kind="mixed", n=32768, nrhs=8, precision="T", kappa=1e6),
        # the same path for data that starts on the host
        dict(name="mixed_host_16384", kind="host", n=16384, nrhs=8, precision="T", kappa=1e2),
        # thousands of uneven matrices in one launch, both precisions
        dict(name="batched_d_4096", kind="batched", type="d", count=4096, lo=16, hi=512),
        dict(name="batched_s_4096", kind="batched", type="s", count=4096, lo=16, hi=512),
        # one step of a Gaussian-process fit: a batch of problems, and one large problem
        dict(name="gp_d_256x1024", kind="gp", type="d", batch=256, n=1024, dim=2, shared=True),
        dict(name="gp_s_1x16384", kind="gp", type="s", batch=1, n=16384, dim=2, shared=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["posv", "posv", "posv", "mixed", "host", "batched", "gp", "gp"])
    if kind == "posv":
        t = rng.choice("dddzsc")
        return dict(kind=kind, type=t, uplo=rng.choice("LLLU"), n=_log(rng, 64, 8192 if t in "zc" else 16384),
                    nrhs=_log(rng, 1, 64), pad=rng.choice([0, 0, 1, 6, 16]),
                    matrix=rng.choice(["gram", "se"]) if t in "dz" else "gram", split=rng.random() < 0.4)
    if kind in ("mixed", "host"):
        precision = rng.choice("TTB")
        return dict(kind=kind, n=_log(rng, 2048, 32768 if kind == "mixed" else 16384), nrhs=rng.randint(1, 8),
                    precision=precision, kappa=10.0 ** rng.randint(1, 6 if precision == "T" and kind == "mixed" else 3))
    if kind == "batched":
        hi = _log(rng, 64, 512)
        return dict(kind=kind, type=rng.choice("ds"), count=_log(rng, 256, 4096), lo=max(1, hi // rng.choice([2, 8, 32])),
                    hi=hi)
    if rng.random() < 0.3:
        return dict(kind="gp", type="s", batch=1, n=_log(rng, 2048, 16384), dim=2, shared=True)
    n = _log(rng, 64, 1024)
    return dict(kind="gp", type=rng.choice("dds"), batch=max(1, min(_log(rng, 8, 512), int(256 * 1024 ** 3 / n ** 3))),
                n=n, dim=rng.randint(1, 3), shared=rng.random() < 0.5)


# ---- inputs ---------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _posv_matrix(case, seed):
    """The Hermitian matrix of a posv case, row-major."""
    n, dt = case["n"], TORCH[case["type"]]
    if case["matrix"] == "se":
        return se_kernel(n, seed, complex_=dt.is_complex, device=DEV).to(dt)
    g = torch.randn(n, n, generator=_generator(seed), device=DEV, dtype=dt)
    a = g @ g.conj().T / n
    a.diagonal().add_(1.0)
    return a


def _posv_rhs(case, seed):
    return torch.randn(case["nrhs"], case["n"], generator=_generator(seed + 7919), device=DEV, dtype=TORCH[case["type"]])


def _posv_storage(case, seed):
    """Column-major storage of the matrix (row j of the tensor is column j), padded leading dimension."""
    a = _posv_matrix(case, seed)
    buf = torch.zeros(case["n"], case["n"] + case["pad"], dtype=a.dtype, device=DEV)
    buf[:, :case["n"]] = a.T
    return buf


def _orders(case):
    """The orders belong to the case, like the sizes of the others; the seed changes the matrices."""
    return np.random.default_rng(0xDD1A0004 + case["count"]).integers(case["lo"], case["hi"] + 1, size=case["count"]).astype(np.int32)


def _batch(case, seed):
    """(orders, matrix offsets, vector offsets, matrices, right-hand sides): A_i = G_i G_i^T / n_i + 0.1 I, packed."""
    orders = _orders(case)
    big = orders.astype(np.int64)
    sizes, lens = (big * big + 31) // 32 * 32, (big + 31) // 32 * 32
    a_off, b_off = np.cumsum(sizes) - sizes, np.cumsum(lens) - lens
    dt, g = TORCH[case["type"]], _generator(seed)
    mats = torch.zeros(int(sizes.sum()), dtype=dt, device=DEV)
    rhs = torch.randn(int(lens.sum()), generator=g, dtype=dt, device=DEV)
    for n in np.unique(orders):
        idx = np.nonzero(orders == n)[0]
        n = int(n)
        w = torch.randn(len(idx), n, n, generator=g, device=DEV, dtype=torch.float64)
        m = torch.baddbmm(0.1 * torch.eye(n, device=DEV, dtype=torch.float64), w, w.mT, alpha=1.0 / n).to(dt)
        at = torch.from_numpy(a_off[idx]).to(DEV)[:, None] + torch.arange(n * n, device=DEV)
        mats[at] = m.reshape(len(idx), n * n)
    return orders, a_off, b_off, mats, rhs


def _gp_inputs(case, seed):
    """Points uniform in the unit cube, y ~ N(0, 1), theta = (lengthscale, signal variance, noise variance)."""
    g, dt = _generator(seed), TORCH[case["type"]]
    b, n = case["batch"], case["n"]
    x = torch.rand(b, n, case["dim"], generator=g, device=DEV, dtype=torch.float64).to(dt)
    y = torch.randn(b, n, generator=g, device=DEV, dtype=torch.float64).to(dt)
    theta = torch.tensor([0.3, 1.0, 1e-2], dtype=torch.float64, device=DEV)
    if not case["shared"]:
        theta = theta * (1.0 + 0.2 * torch.rand(b, 3, generator=g, device=DEV, dtype=torch.float64))
    return x, y, theta


# ---- what is measured -----------------------------------------------------------------


def prepare(case, seed):
    handle = autograd.default_handle()
    state = dict(case=case, handle=handle)
    kind = case["kind"]
    if kind == "posv":
        n, nrhs, lld, dt = case["n"], case["nrhs"], case["n"] + case["pad"], NUMPY[case["type"]]
        a, b = _posv_storage(case, seed), _posv_rhs(case, seed)
        fa, x = torch.zeros_like(a), torch.zeros_like(b)
        wrap = ddla.DistributedMatrix.wrap
        state.update(a=a, b=b, fa=fa, x=x, a_bytes=a.numel() * a.element_size(), b_bytes=b.numel() * b.element_size(),
                     dA=wrap(handle, fa.data_ptr(), n, n, lld, dt, mb=256, nb=256),
                     dX=wrap(handle, x.data_ptr(), n, nrhs, n, dt, mb=256, nb=256))
    elif kind in ("mixed", "host"):
        n, nrhs = case["n"], case["nrhs"]
        a = householder_spd(n, case["kappa"], seed, device=DEV)
        b = torch.randn(nrhs, n, generator=_generator(seed + 7919), device=DEV, dtype=torch.float64)
        if kind == "host":
            pa, pb = (torch.empty(t.shape, dtype=t.dtype, pin_memory=True) for t in (a, b))
            pa.copy_(a)
            pb.copy_(b)
            px = torch.zeros(nrhs, n, dtype=torch.float64).pin_memory()
            state.update(keep=(pa, pb, px), A=pa.numpy().T, B=pb.numpy().T, X=px.numpy().T)
        else:
            x = torch.zeros_like(b)
            wrap = lambda t, cols: ddla.DistributedMatrix.wrap(handle, t.data_ptr(), n, cols, n, np.float64, mb=256,  # noqa: E731
                                                              nb=256)
            state.update(a=a, b=b, x=x, dA=wrap(a, n), dB=wrap(b, nrhs), dX=wrap(x, nrhs))
    elif kind == "batched":
        orders, a_off, b_off, mats, rhs = _batch(case, seed)
        es = BYTES[case["type"]]
        work, x = torch.zeros_like(mats), torch.zeros_like(rhs)
        up = lambda v, dt: torch.from_numpy(v.astype(dt)).to(DEV)  # noqa: E731
        pb = batched.PackedBatch(dtype=np.dtype(NUMPY[case["type"]]), orders=orders, a_offsets=a_off, b_offsets=b_off,
                                 mats=work, rhs=x, d_n=up(orders, np.int32), d_lda=up(orders, np.int32),
                                 d_A=up(work.data_ptr() + a_off * es, np.int64),
                                 d_B=up(x.data_ptr() + b_off * es, np.int64),
                                 logdet=torch.zeros(len(orders), dtype=torch.float64, device=DEV),
                                 info=torch.zeros(len(orders), dtype=torch.int32, device=DEV), max_n=512)
        torch.cuda.synchronize()
        if case["type"] not in _tuned:  # once per process, as a program that runs such batches does
            batched.autotune(handle, case["type"], 512)
            _tuned.add(case["type"])
        state.update(mats=mats, b=rhs, pb=pb, plan=batched.VbatchedPlan(handle, pb), a_bytes=mats.numel() * es,
                     b_bytes=rhs.numel() * es)
    else:
        x, y, theta = _gp_inputs(case, seed)
        state.update(points=x, y=y, theta=theta.requires_grad_())
    torch.cuda.synchronize()
    return state


def run(state):
    case, handle = state["case"], state["handle"]
    kind = case["kind"]
    if kind == "posv":
        dA, dX = state["dA"], state["dX"]
        handle.memcpy(dA.data_ptr, state["a"].data_ptr(), state["a_bytes"])
        handle.memcpy(dX.data_ptr, state["b"].data_ptr(), state["b_bytes"])
        if not case["split"]:
            _, info = ddla.pposv(dA, dX, uplo=case["uplo"])
            return [state["fa"], state["x"], info]
        _, info = ddla.ppotrf(dA, uplo=case["uplo"])
        ddla.ppotrs(dA, dX, uplo=case["uplo"])
        return [state["fa"], state["x"], info, 2.0 * ddla.diag_logdet(dA).real]
    if kind == "mixed":
        _, info, _ = ddla.pposv_mixed(state["dA"], state["dB"], state["dX"], precision=case["precision"])
        return [state["x"], info]
    if kind == "host":
        _, info, _ = ddla.pposv_mixed_host(handle, state["A"], state["B"], precision=case["precision"], X=state["X"])
        return [state["keep"][2], info]
    if kind == "batched":
        pb = state["pb"]
        handle.memcpy(pb.mats.data_ptr(), state["mats"].data_ptr(), state["a_bytes"])
        handle.memcpy(pb.rhs.data_ptr(), state["b"].data_ptr(), state["b_bytes"])
        state["plan"].run()
        return [pb.mats, pb.rhs, pb.logdet, pb.info]
    loss = autograd.gp_nll(state["points"], state["y"], state["theta"])
    (grad,) = torch.autograd.grad(loss.sum(), state["theta"])
    return [loss, grad]


def work(case):
    kind = case["kind"]
    if kind == "batched":
        x = _orders(case).astype(np.float64)
        es = BYTES[case["type"]]
        return dict(bytes=float((es * (x * (x + 1) + 2 * x)).sum()), flops=float((x ** 3 / 3 + 2 * x * x).sum()))
    n = float(case["n"])
    if kind == "gp":
        # Cholesky, inverse of the factor's triangle, and the product that the gradient contracts: n^3 / 3 each
        return dict(bytes=case["batch"] * n * (case["dim"] + 1) * BYTES[case["type"]], flops=case["batch"] * n ** 3)
    nrhs = case["nrhs"]
    mul = 4 if case.get("type", "d") in "cz" else 1
    es = BYTES[case.get("type", "d")]
    moved = n * (n + 1) / 2 * es * (2 if kind == "posv" else 1) + 2 * n * nrhs * es
    return dict(bytes=moved, flops=mul * (n ** 3 / 3 + 2 * n * n * nrhs))


def tolerance(case):
    # measured against exact() over the ranges above, four to eight times the largest seen
    kind = case["kind"]
    if kind == "posv":
        if case["type"] in "sc":
            return dict(rel=1.2e-5, max=1e-4)
        # the kernel matrices have condition numbers up to about 1e5, the Gram matrices about 5
        return dict(rel=4e-11, max=4e-10) if case["matrix"] == "se" else dict(rel=4e-14, max=4e-13)
    if kind in ("mixed", "host"):
        # refinement stops at a normwise backward error of eps sqrt(n): kappa times that in the solution
        return dict(rel=2.5e-14 * case["kappa"] + 2e-14, max=min(0.5, 5e-13 * case["kappa"] + 1e-12))
    if kind == "batched":
        return dict(rel=1e-5, max=1e-4) if case["type"] == "s" else dict(rel=2e-14, max=1e-13)
    return dict(rel=7e-4, max=7e-4) if case["type"] == "s" else dict(rel=4e-13, max=8e-13)


# ---- the same results in 64 bits ------------------------------------------------------


def _wide(t):
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def _factor_into(storage, a, uplo):
    """The factor of row-major Hermitian `a` written over the chosen triangle of its column-major storage."""
    n = a.shape[0]
    low = torch.linalg.cholesky(a)
    view = storage[:, :n]
    # storage is the transpose: its upper part holds the lower triangle of the matrix
    tri = low.T if uplo == "L" else low.conj()
    mask = torch.ones(n, n, dtype=torch.bool, device=DEV)
    mask = mask.triu() if uplo == "L" else mask.tril()
    view[mask] = tri[mask]
    return low


def _gp_exact(x, y, theta):
    n = x.shape[0]
    ell, sf, noise = (float(v) for v in theta)
    d2 = sum((x[:, None, k] - x[None, :, k]) ** 2 for k in range(x.shape[1]))
    k = sf * torch.exp(-d2 / (2 * ell * ell))
    low = torch.linalg.cholesky(k + noise * torch.eye(n, dtype=torch.float64, device=DEV))
    alpha = torch.cholesky_solve(y[:, None], low)[:, 0]
    loss = 0.5 * (y @ alpha) + torch.log(low.diagonal()).sum()
    g = torch.cholesky_inverse(low)
    g -= alpha[:, None] * alpha[None, :]
    g *= 0.5
    noise_part = g.diagonal().sum()
    g *= k
    return loss, torch.stack([(g * d2).sum() / ell ** 3, g.sum() / sf, noise_part])


def exact(case, seed):
    kind = case["kind"]
    if kind == "posv":
        storage, b = _wide(_posv_storage(case, seed)), _wide(_posv_rhs(case, seed))
        a = storage[:, :case["n"]].T.contiguous()
        low = _factor_into(storage, a, case["uplo"])
        x = torch.cholesky_solve(b.T.contiguous(), low).T.contiguous()
        out = [storage, x, 0]
        return out + [2.0 * float(low.diagonal().real.log().sum())] if case["split"] else out
    if kind in ("mixed", "host"):
        a = householder_spd(case["n"], case["kappa"], seed, device=DEV)
        b = torch.randn(case["nrhs"], case["n"], generator=_generator(seed + 7919), device=DEV, dtype=torch.float64)
        x = torch.cholesky_solve(b.T.contiguous(), torch.linalg.cholesky(a)).T.contiguous()
        return [x.cpu() if kind == "host" else x, 0]
    if kind == "batched":
        orders, a_off, b_off, mats, rhs = _batch(case, seed)
        mats, rhs = _wide(mats), _wide(rhs)
        logdet = torch.zeros(len(orders), dtype=torch.float64, device=DEV)
        for i, n in enumerate(int(v) for v in orders):
            storage = mats[a_off[i]:a_off[i] + n * n].view(n, n)
            low = torch.linalg.cholesky(storage.T)
            v = rhs[b_off[i]:b_off[i] + n]
            v.copy_(torch.cholesky_solve(v[:, None], low)[:, 0])
            logdet[i] = 2.0 * low.diagonal().log().sum()
            storage.copy_(torch.tril(storage, -1) + low.T)
        return [mats, rhs, logdet, None]
    x, y, theta = _gp_inputs(case, seed)
    x, y = x.double(), y.double()
    one = [_gp_exact(x[i], y[i], theta if case["shared"] else theta[i]) for i in range(case["batch"])]
    loss, grad = torch.stack([o[0] for o in one]), torch.stack([o[1] for o in one])
    return [loss, grad.sum(0) if case["shared"] else grad]
