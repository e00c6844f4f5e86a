"""The workloads by which the speed of this framework is judged, one pass of each through the
public entry points of ``crava_b200.api``.

A case is a dict of plain values.  ``op`` says which calls a pass makes:

  run     Job.run on a block whose inputs are resident: the inversion itself (posterior mean,
          posterior covariance and ``sims`` conditional realisations).  ``prior`` "factors" is
          the separable prior, "grids" the prior grids generated on the device by
          Job.fill_prior with the correlation gradients of a dipping block, each pass;
          ``thick`` a block of non-constant thickness (Job.divide_data before the run, on data
          put back each pass, because the division works in place); ``resid`` keeps the
          residual spectra; ``fp64`` is the threshold of the FP64 re-factorisation.
  host    api.invert_block on host buffers: job creation, uploads, run and downloads.
  batch   api.Batch.run: several blocks of uneven size and angle count as one graph.
  fft     api.fft_r2c and api.fft_c2r of one device grid (FFTGrid::fftInPlace / invFFTInPlace).
  facies  api.facies_smooth of the facies histograms and api.facies_prob on a posterior mean.

Sizes, angle stacks, wavelets and priors are those of the benchmark's blocks
(crava_b200/synth.py, bench.py) and of the tests; the data are white noise of seismic
amplitude, as in the benchmark's throughput runs.
"""
import math
import random

import numpy as np
import torch

from crava_b200 import api, synth


def _smooth(lo, hi):
    """2,3,5,7-smooth lengths in [lo, hi], the sizes a padded grid can have."""
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


def _run(name, nx, ny, nz, angles, sims, **more):
    c = {"name": name, "op": "run", "nx": nx, "ny": ny, "nz": nz, "angles": angles, "sims": sims, "prior": "factors",
         "thick": False, "resid": False, "fp64": 0.0, "wide": False}
    c.update(more)
    return c


def listed():
    return [
        # a test-sized block: launches and latency are all of it
        _run("tiny 32x30x40", 32, 30, 40, 2, 1),
        # the CPU-runnable block of the benchmark suite
        _run("small 64x64x128", 64, 64, 128, 3, 1),
        # one block of the mixed batch: odd lengths in all three directions, 16 realisations
        _run("odd 105x135x125", 105, 135, 125, 4, 16),
        # an ordinary block whose lengths are not the tuned ones (bench.py --kernels)
        _run("general 250x250x200", 250, 250, 200, 5, 4),
        # the production block
        _run("production 540x540x256", 540, 540, 256, 5, 4),
        # the precision-study block: the largest, six angles and a wide band
        _run("largest 768x768x320", 768, 768, 320, 6, 1, wide=True),
        # dipping correlation: prior grids instead of factors, FP64 re-factorisation on
        _run("grids 200x216x200", 200, 216, 200, 3, 2, prior="grids", fp64=100.0),
        # non-constant thickness, residuals kept for the synthetics
        _run("thick 270x270x256", 270, 270, 256, 5, 4, thick=True, resid=True),
        # host to host, as a program that inverts one block and leaves
        {"name": "host 64x64x128", "op": "host", "nx": 64, "ny": 64, "nz": 128, "angles": 3, "sims": 1, "wide": False},
        # uneven blocks of the mixed batch, 2..6 angles, 16 realisations, as one graph
        {"name": "batch of 12", "op": "batch", "blocks": 12, "shapes": 7, "sims": 16, "wide": False},
        # one grid there and back
        {"name": "fft 540x540x256", "op": "fft", "nx": 540, "ny": 540, "nz": 256, "covariance": False},
        # facies probabilities of a posterior mean, 100x100x50 density volumes
        {"name": "facies 270x270x256", "op": "facies", "nx": 270, "ny": 270, "nz": 256, "facies": 3,
         "bins": 100},
    ]


def draw(rng):
    op = rng.choice(["run"] * 7 + ["host", "batch", "fft", "fft", "facies"])
    top = {"run": 4e7, "host": 1.2e6, "fft": 7e7, "facies": 2e7, "batch": 0}[op]
    if op == "batch":
        return {"op": "batch", "blocks": rng.randint(4, 12), "shapes": rng.randrange(1000), "sims": rng.randint(1, 16),
                "wide": rng.random() < 0.5}
    low = {"run": 3e4, "host": 1e5, "fft": 1e5, "facies": 2e5}[op]
    lateral, depth = _smooth(16, 768), _smooth(40, 320)
    want = math.exp(rng.uniform(math.log(low), math.log(top)))
    nz = min(depth, key=lambda n: abs(n - want ** (1 / 3) * rng.uniform(0.6, 1.6)))
    side = math.sqrt(want / nz)
    f = rng.uniform(0.7, 1.4)
    nx = min(lateral, key=lambda n: abs(n - side * f))
    ny = min(lateral, key=lambda n: abs(n - side / f))
    if op == "fft":
        return {"op": "fft", "nx": nx, "ny": ny, "nz": nz, "covariance": rng.random() < 0.5}
    if op == "facies":
        return {"op": "facies", "nx": nx, "ny": ny, "nz": nz, "facies": rng.randint(2, 4),
                "bins": rng.choice([40, 64, 80, 100])}
    angles = rng.randint(1, 6)
    sims = rng.choice([0, 1, 1, 2, 4, 8, 16])
    c = {"op": op, "nx": nx, "ny": ny, "nz": nz, "angles": angles, "sims": sims, "wide": rng.random() < 0.3}
    if op == "run":
        kind = rng.choice(["plain"] * 4 + ["grids", "thick", "fp64", "resid"])
        c.update(prior="grids" if kind == "grids" else "factors", thick=kind == "thick",
                 resid=kind == "resid", fp64=100.0 if kind == "fp64" else 0.0)
    return c


# ------------------------------------------------------------------ the block of a case

GRAD = (0.3, -0.2)          # correlation gradients of the "grids" prior, samples per trace
PAIRS = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
MEAN = (math.log(3000.0), math.log(1500.0), math.log(2300.0))
DT = 4.0                    # ms
AMP = 0.02                  # amplitude of the seismic


def _model(case, seed):
    """What describes a block beside its grids, as numpy arrays in the reference's
    representation: priors within 30 % of the benchmark's, one 25..35 Hz Ricker per angle."""
    r = np.random.RandomState(int(seed) % (1 << 31))
    nx, ny, nz, n = case["nx"], case["ny"], case["nz"], case["angles"]
    f4 = lambda a: np.asarray(a, np.float64).astype(np.float32)  # noqa: E731
    low, high = (2.0, 120.0) if case["wide"] else (5.0, 55.0)
    th = np.deg2rad(np.linspace(5.0, 50.0 if case["wide"] else 45.0, n) if n > 1 else np.array([20.0]))
    th = f4(th).astype(np.float64)
    s2, t2 = np.sin(th) ** 2, np.tan(th) ** 2
    A = f4(np.stack([(1 + t2) / 2, -s2, (1 - s2) / 2], axis=1)).astype(np.float64)
    sd = np.array([0.08, 0.15, 0.05]) * r.uniform(0.7, 1.3, 3)
    C = np.eye(3)
    C[0, 1] = C[1, 0] = 0.7 * r.uniform(0.8, 1.2)
    C[0, 2] = C[2, 0] = 0.5 * r.uniform(0.8, 1.2)
    C[1, 2] = C[2, 1] = 0.4 * r.uniform(0.8, 1.2)
    pv = f4(sd[:, None] * sd[None, :] * C).astype(np.float64)
    # spherical lateral correlation, 25 m cells
    rng_m = 1000.0 * r.uniform(0.7, 1.3)
    i, j = np.arange(nx), np.arange(ny)
    di = np.where(i < nx // 2 + 1, i, i - nx) * 25.0 / rng_m
    dj = np.where(j < ny // 2 + 1, j, j - ny) * 25.0 / rng_m
    d = np.sqrt(di[None, :] ** 2 + dj[:, None] ** 2)
    cxy = f4(np.where(d >= 1, 0.0, 1 + d ** 3 / 2 - 1.5 * d))
    # circular Gaussian temporal correlation, the spectrum zeroed at and below low_cut
    k = np.arange(nz)
    lag = np.minimum(k, nz - k)
    F = np.abs(np.fft.rfft(f4(np.exp(-3.0 * (DT * lag / 40.0) ** 2)).astype(np.float64)))
    F[: int(math.floor(low * (nz * 0.001 * DT))) + 1] = 0.0
    back = np.fft.irfft(F, n=nz)
    cct = f4(back / back[0])
    z = np.where(k < nz // 2 + 1, DT * k, DT * (k - nz))
    wav = []
    for p in (np.linspace(25.0, 35.0, n) if n > 1 else [30.0]):
        c = (math.pi * p * z) ** 2 * 1e-6
        wav.append(np.where(np.abs(z) <= 119.0, (1 - 2 * c) * np.exp(-c), 0.0))
    wav = f4(wav)
    wn = f4(np.sqrt((wav.astype(np.float64) ** 2).sum(axis=1)))
    sn = np.linspace(2.0, 10.0, n) if case["wide"] else np.full(n, 5.0)
    ev = AMP ** 2 / sn
    deg = np.rad2deg(th)
    ang = np.exp(-3.0 * np.abs(deg[:, None] - deg[None, :]) / 10.0)
    etc = f4(np.sqrt(ev[:, None] * ev[None, :]) * ang).astype(np.float64)
    m = dict(A=A, etc=etc, wav=wav, wn=wn, pv=pv, cxy=cxy, cct=cct, low=low, high=high, wnc=0.1, lz=nz * DT, rt=None,
             min_rt=1.0)
    if case.get("thick"):
        x, y = np.arange(nx)[None, :] / nx, np.arange(ny)[:, None] / ny
        a, b = r.uniform(0, 2 * np.pi, 2)
        rt = 0.75 + 0.55 * (0.5 + 0.25 * np.sin(2 * np.pi * x + a) + 0.25 * np.cos(3 * np.pi * y + b))
        m["rt"] = f4(rt).astype(np.float64)
        m["min_rt"] = float(m["rt"].min())
    return m


def _block(case, m):
    """The block description that the binding takes; its grids stay on the device."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return synth.Block(spec=None, nx=nx, ny=ny, nz=nz, nxp=nx, nyp=ny, nzp=nz, lz=m["lz"], A=m["A"],
                       err_theta_cov=m["etc"], wavelet=m["wav"], wavelet_norm=m["wn"], prior_var0=m["pv"],
                       corr_xy=m["cxy"], prior_corr_t=None, circ_corr_t=m["cct"], low_int_cut=0, mean=None, data=None,
                       low_cut=m["low"], high_cut=m["high"], wnc=m["wnc"], min_rel_thick=m["min_rt"],
                       nsim=case["sims"], seed=0, rel_thick=m["rt"])


def _fill(out, nx, seed, l, mean=None):
    """Seeded values of one input grid (nz, ny, row): noise of seismic amplitude, or a prior mean
    with a gentle trend in depth and a little lateral variation."""
    g = torch.Generator("cuda").manual_seed((int(seed) * 64 + l) % (1 << 62))
    nz, ny = out.shape[0], out.shape[1]
    out[..., nx:] = 0
    if mean is None:
        out[..., :nx] = torch.randn((nz, ny, nx), generator=g, device="cuda") * AMP
    else:
        z = torch.linspace(-0.05, 0.05, nz, device="cuda")[:, None, None]
        lat = torch.randn((1, ny, nx), generator=g, device="cuda") * 0.01
        out[..., :nx] = mean + z + lat


_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = api.Context(torch.cuda.current_device())
    return _ctx


class _Memory:
    """Device memory of a job, as torch takes it; it keeps the job alive."""

    def __init__(self, job, ptr, shape, strides=None, typestr="<f4"):
        self.job = job
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": strides}


def _grids(job, role, count, complex_=False):
    """The job's `count` grids of a role as one tensor: (count, nz, ny, nx), or (count, nz, ny,
    cnx) complex spectra."""
    nz, ny, row = job.shape
    p = [job.device_ptr(role, i) for i in range(count)]
    step = p[1] - p[0] if count > 1 else 4 * nz * ny * row
    assert all(p[i] == p[0] + i * step for i in range(count))
    if complex_:
        return torch.as_tensor(_Memory(job, p[0], (count, nz, ny, row // 2), (step, 4 * ny * row, 4 * row, 8), "<c8"),
                               device="cuda")
    return torch.as_tensor(_Memory(job, p[0], (count, nz, ny, row), (step, 4 * ny * row, 4 * row, 4)), device="cuda")


def _job(case, seed):
    """A created job with its inputs on the device, and its outputs as tensors."""
    m = _model(case, seed)
    blk = _block(case, m)
    flags = api.FLAG_KEEP_RESIDUAL if case.get("resid") else 0
    prior = api.PRIOR_GRIDS if case.get("prior") == "grids" else api.PRIOR_SEPARABLE
    job = api.Job(_context(), blk, prior, flags, seed=seed, fp64_threshold=case.get("fp64", 0.0))
    nx = case["nx"]
    data, mean = _grids(job, api.ROLE_DATA, blk.ntheta), _grids(job, api.ROLE_MEAN, 3)
    for l in range(blk.ntheta):
        _fill(data[l], nx, seed, l)
    for a in range(3):
        _fill(mean[a], nx, seed, 16 + a, MEAN[a])
    out = {"mean": _grids(job, api.ROLE_POST_MEAN, 3)[..., :nx], "cov": _grids(job, api.ROLE_POST_COV, 6)[..., :nx]}
    if case["sims"]:
        out["sims"] = _grids(job, api.ROLE_SIM, 3 * case["sims"])[..., :nx]
    if case.get("resid"):
        out["resid"] = _grids(job, api.ROLE_RESIDUAL, blk.ntheta, True)
    return job, data, out


def _batch_cases(case):
    r = random.Random(case["shapes"])
    xy, zz = _smooth(64, 256), _smooth(64, 200)
    return [{"op": "run", "nx": r.choice(xy), "ny": r.choice(xy), "nz": r.choice(zz), "angles": r.randint(2, 6),
             "sims": case["sims"], "wide": case["wide"]} for _ in range(case["blocks"])]


def _facies_model(case, seed):
    r = np.random.RandomState(int(seed) % (1 << 31))
    nb = (case["bins"], case["bins"], case["bins"] // 2)
    vmin = [MEAN[0] - 0.35, MEAN[1] - 0.6, MEAN[2] - 0.25]
    dv = [0.7 / nb[0], 1.2 / nb[1], 0.5 / nb[2]]
    prior = r.uniform(0.5, 1.5, case["facies"])
    sig = np.array([[0.003, 0.001, 0.0005], [0.001, 0.004, 0.0002], [0.0005, 0.0002, 0.001]]) * r.uniform(0.5, 2)
    # histograms of well samples around each facies' centre
    hist = np.zeros((case["facies"], nb[2], nb[1], nb[0]))
    for f in range(case["facies"]):
        c = [r.uniform(0.3, 0.7) * n for n in nb]
        at = [np.clip((c[d] + r.standard_normal(300) * nb[d] * 0.08).astype(int), 0, nb[d] - 1) for d in range(3)]
        np.add.at(hist[f], (at[2], at[1], at[0]), 1.0 / 300)
    return dict(nb=nb, vmin=vmin, dv=dv, prior=(prior / prior.sum()).astype(np.float32), undef=0.02,
                sinv=np.linalg.inv(sig), hist=hist.astype(np.float32))


def _facies_mean(case, seed):
    """A posterior mean: three smooth fields about the background, (3, nz, ny, row)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    out = torch.zeros((3, nz, ny, 2 * (nx // 2 + 1)), device="cuda")
    ph = np.random.RandomState((int(seed) + 1) % (1 << 31)).uniform(0, 2 * np.pi, (3, 3))
    g = torch.Generator("cuda").manual_seed(int(seed) % (1 << 62))
    ax = [torch.arange(n, device="cuda") / n for n in (nz, ny, nx)]
    for a, s in enumerate((0.08, 0.15, 0.05)):
        f = torch.sin(40 * ax[0] + ph[a, 0])[:, None, None] + torch.sin(9 * ax[1] + ph[a, 1])[None, :, None] \
            + torch.cos(12 * ax[2] + ph[a, 2])[None, None, :]
        out[a, ..., :nx] = MEAN[a] + s * (0.7 * f + 0.3 * torch.randn((nz, ny, nx), generator=g, device="cuda"))
    return out


# ------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    seed = int(seed)
    op = case["op"]
    if op == "run":
        job, data, out = _job(case, seed)
        s = {"op": op, "job": job, "out": out, "grids": case["prior"] == "grids", "thick": case["thick"], "data": data}
        if case["thick"]:
            s["seismic"] = data.clone()
        return s
    if op == "host":
        m = _model(case, seed)
        blk = _block(case, m)
        row = 2 * (case["nx"] // 2 + 1)
        buf = torch.empty((blk.ntheta + 3, case["nz"], case["ny"], row), device="cuda")
        for l in range(blk.ntheta + 3):
            _fill(buf[l], case["nx"], seed, l if l < blk.ntheta else 16 + l - blk.ntheta,
                  None if l < blk.ntheta else MEAN[l - blk.ntheta])
        h = buf.cpu().numpy()
        blk.data, blk.mean = h[:blk.ntheta], h[blk.ntheta:]
        return {"op": op, "ctx": _context(), "blk": blk, "seed": seed, "nx": case["nx"]}
    if op == "batch":
        jobs = [_job(c, seed * 16 + i) for i, c in enumerate(_batch_cases(case))]
        return {"op": op, "batch": api.Batch(_context(), [j[0] for j in jobs], branches=1), "out": [j[2] for j in jobs]}
    if op == "fft":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        x = torch.empty((nz, ny, 2 * (nx // 2 + 1)), device="cuda")
        _fill(x, nx, seed, 0)
        return {"op": op, "ctx": _context(), "x": x, "spec": torch.empty_like(x), "back": torch.empty_like(x),
                "dims": (nx, ny, nz), "cov": case["covariance"]}
    m = _facies_model(case, seed)
    nb, nx, ny, nz = m["nb"], case["nx"], case["ny"], case["nz"]
    fd, keep = api.facies_desc(m["prior"], nb, m["vmin"], m["dv"], m["undef"])
    hist = torch.zeros((case["facies"], nb[2], nb[1], 2 * (nb[0] // 2 + 1)), device="cuda")
    hist[..., :nb[0]] = torch.from_numpy(m["hist"]).cuda()
    return {"op": op, "ctx": _context(), "fd": fd, "keep": keep, "sinv": m["sinv"], "hist": hist,
            "dens": torch.empty_like(hist), "bins": nb, "mean": _facies_mean(case, seed), "dims": (nx, ny, nz),
            "prob": torch.empty((case["facies"] + 1, nz, ny, 2 * (nx // 2 + 1)), device="cuda")}


def run(s):
    op = s["op"]
    if op == "run":
        if s["grids"]:
            s["job"].fill_prior(*GRAD)
        if s["thick"]:
            s["data"].copy_(s["seismic"])
            s["job"].divide_data()
        s["job"].run()
        return s["out"]
    if op == "host":
        out = api.invert_block(s["ctx"], s["blk"], seed=s["seed"])
        return {k: out[k][..., :s["nx"]] for k in ("mean", "cov", "sims") if k in out}
    if op == "batch":
        s["batch"].run()
        return s["out"]
    if op == "fft":
        nx, ny, nz = s["dims"]
        s["spec"].copy_(s["x"])
        api.fft_r2c(s["ctx"], s["spec"].data_ptr(), nx, ny, nz, s["cov"])
        s["back"].copy_(s["spec"])
        api.fft_c2r(s["ctx"], s["back"].data_ptr(), nx, ny, nz, s["cov"])
        return {"spec": s["spec"], "back": s["back"][..., :nx]}
    nx, ny, nz = s["dims"]
    s["dens"].copy_(s["hist"])
    api.facies_smooth(s["ctx"], s["fd"], s["sinv"], s["dens"].data_ptr())
    api.facies_prob(s["ctx"], s["fd"], s["dens"].data_ptr(), s["dens"].shape[3], [t.data_ptr() for t in s["mean"]], nx, ny,
                    nz, nx, ny, [t.data_ptr() for t in s["prob"]])
    return {"dens": s["dens"][..., :s["bins"][0]], "prob": s["prob"][..., :nx]}


def work(case):
    op = case["op"]
    if op == "batch":
        w = [work(c) for c in _batch_cases(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    N = case["nx"] * case["ny"] * case["nz"]
    fft = 2.5 * N * math.log2(N)
    if op == "fft":
        return {"bytes": 4.0 * 3 * N, "flops": 2 * fft}
    if op == "facies":
        nb = case["bins"] ** 2 * (case["bins"] // 2)
        f = case["facies"]
        return {"bytes": 4.0 * (N * (3 + f + 1) + 2 * nb * f),
                "flops": N * (20.0 + 16 * f) + (2 * f + 1) * 2.5 * nb * math.log2(nb)}
    n, s = case["angles"], case["sims"]
    grids = n + 3 + 9 + 3 * s + (n if case.get("resid") else 0)
    # transforms, then per bin of the half spectrum the data system, its solves and the draws
    per_bin = 8.0 * (n * n + 12 * n) + 60 + s * 100
    return {"bytes": 4.0 * N * grids, "flops": fft * grids + N / 2 * per_bin}


# ------------------------------------------------------------------ the same in 64 bits

def _philox(c0, c1, s, seed):
    """The counter-based noise words of bins (c1, c0) of realisation s: Philox-4x32, 7 rounds, in
    64-bit integers."""
    M = 0xFFFFFFFF

    def mul(a, b):     # 32 x 32 -> (high, low), a constant
        bl, bh = b & 0xFFFF, b >> 16
        p0, p1 = a * bl, a * bh                     # < 2^48
        lo = p0 + ((p1 & 0xFFFF) << 16)
        return (p1 >> 16) + (lo >> 32), lo & M

    x, y, z, w = c0, c1, torch.full_like(c0, s), torch.zeros_like(c0)
    kx, ky = seed & M, (seed >> 32) & M
    for _ in range(7):
        h0, l0 = mul(0xD2511F53, x)
        h1, l1 = mul(0xCD9E8D57, z)
        x, y, z, w = h1 ^ y ^ kx, l1, h0 ^ w ^ ky, l0
        kx, ky = (kx + 0x9E3779B9) & M, (ky + 0xBB67AE85) & M
    return x, y, z, w


def _noise(seed, s, k, ny, nz, nx):
    """Three complex normals per bin of the planes k (1-D tensor): list of (len(k), ny, cnx)."""
    cn = nx // 2 + 1
    dev = "cuda"
    K = k[:, None, None]
    J = torch.arange(ny, device=dev)[None, :, None]
    I = torch.arange(cn, device=dev)[None, None, :]
    plane = (I == 0) | ((nx % 2 == 0) & (I == cn - 1))
    jc, kc = torch.where(J == 0, J, ny - J), torch.where(K == 0, K, nz - K)
    a, b = J + ny * K, jc + ny * kc
    me = plane & (a == b)
    cj = plane & (b < a)
    bin_ = (torch.where(cj, kc, K) * ny + torch.where(cj, jc, J)) * cn + I
    x, y, z, w = _philox(bin_ & 0xFFFFFFFF, bin_ >> 32, s, seed)
    words = [(x >> 6, w & 0xFFFF), (y >> 6, w >> 16), (z >> 6, (x & 63) | ((y & 63) << 6) | ((z & 15) << 12))]
    out = []
    for u, v in words:
        rad = torch.sqrt(-2.0 * torch.log((u.double() + 0.5) / 2 ** 26))
        ang = 2 * math.pi * ((v.double() + 0.5) / 65536 - 0.5)
        re, im = rad * torch.cos(ang), rad * torch.sin(ang)
        h = math.sqrt(0.5)
        im = torch.where(cj, -im, im) * h
        out.append(torch.complex(torch.where(me, re, re * h), torch.where(me, torch.zeros_like(im), im)))
    return out


def _chol(M):
    """Cholesky factor of Hermitian matrices given as lists of tensors, and where it exists (a
    pivot above 1e-20 of the first one)."""
    n = len(M)
    L = [[None] * n for _ in range(n)]
    f = M[0][0].real
    ok = f > 0
    for i in range(n):
        ok = ok & (M[i][i].real > 1e-20 * f)
        for j in range(i + 1):
            s = M[i][j]
            for q in range(j):
                s = s - L[i][q] * L[j][q].conj()
            if i > j:
                L[i][j] = s / L[j][j]
            else:
                ok = ok & (s.real > 1e-20 * f)
                L[i][i] = torch.sqrt(torch.where(ok, s.real, torch.ones_like(s.real)))
    return L, ok


def _solve(L, b):
    n = len(L)
    y = []
    for i in range(n):
        s = b[i]
        for q in range(i):
            s = s - L[i][q] * y[q]
        y.append(s / L[i][i])
    x = [None] * n
    for i in reversed(range(n)):
        s = y[i]
        for q in range(i + 1, n):
            s = s - L[q][i].conj() * x[q]
        x[i] = s / L[i][i]
    return x


def _diff3(w):
    """central(backward(forward)) difference of a wavelet, cyclic."""
    f = np.roll(w, -1) - w
    b = f - np.roll(f, 1)
    return 0.5 * (np.roll(b, -1) - np.roll(b, 1))


def _interp(c, om, scale):
    """The half spectrum c (numpy) stretched: linear interpolation at om, over scale (torch)."""
    t = torch.from_numpy(np.ascontiguousarray(c)).cuda()
    cn = t.numel()
    lo = torch.floor(om).clamp(0, cn - 1)
    d = om - lo
    lo = lo.long()
    hi = (lo + 1).clamp(max=cn - 1)
    return torch.where(om < cn, t[lo] * (1 - d) + t[hi] * d, torch.zeros_like(t[lo])) / scale


def _divide(case, m, data, l):
    """The data of angle l divided by the stretched wavelet, per trace (non-constant thickness)."""
    n = case["nz"]
    cn = n // 2 + 1
    w = m["wav"][l].astype(np.float64)
    W = np.fft.fft(w)[:cn]
    E = np.fft.fft(_diff3(w))[:cn]
    df = 1000.0 / (n * DT)
    lo, hi = max(0, int(math.floor(m["low"] / df))), min(cn, int(math.ceil(m["high"] / df)))
    e2 = 2.0 / n * (np.abs(E[lo:hi]) ** 2).sum() - (np.abs(E[0]) ** 2 / n if lo == 0 else 0.0)
    E = E / math.sqrt(e2)
    a = m["A"][l]
    rc = float(a @ m["pv"] @ a) * m["cct"].astype(np.float64) / float(m["cct"][0])
    rc = 2 * rc - np.roll(rc, -1) - np.roll(rc, 1)
    tau = torch.from_numpy(np.abs(np.fft.fft(rc)[:cn].real)).cuda()[:, None, None]
    wn2 = float(m["wn"][l]) ** 2
    mod = wn2 * ((n // 2) * 1000.0 / (DT * n) / m["high"])
    ev, wnc = m["etc"][l, l], m["wnc"]
    sf = torch.from_numpy(m["rt"]).cuda()[None]
    k = torch.arange(cn, device="cuda", dtype=torch.float64)[:, None, None]
    col = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()[:, None, None]  # noqa: E731
    wl, el = _interp(W, k / sf, sf), _interp(E, k / sf, sf)
    wL, wG = wl.abs() ** 2, col(np.abs(W) ** 2)
    c = (1 - wnc) / 2
    sL = ev * (wnc + c * (wL / wn2 + el.abs() ** 2))
    sG = ev * (wnc + c * (wG / wn2 + col(np.abs(E) ** 2)))
    tm = 0.05 * mod
    gA = torch.where(wG < tm, 0.5 * (wG + tm), wG)
    lA = torch.where(wL < tm, 0.5 * (wL + tm), wL)
    tg = (0.05 * gA).expand_as(lA)
    few = lA < tg
    lA = torch.where(few, 0.5 * (wL + tg), lA)
    sL = torch.where(few, sL * (lA / wL), sL)
    fac = (wl / (tau * lA + sL)) / (gA / (tau * wG + sG))
    freq = k * (1000.0 / (sf * DT * n))
    band = (freq > m["low"]) & (freq < m["high"])
    spec = torch.fft.rfft(data, dim=0)
    return torch.fft.irfft(torch.where(band, spec * fac, torch.zeros_like(fac)), n=n, dim=0)


def _kz(case, m):
    """Per kz and angle: the wavelet and error operators, the white-noise term and the band."""
    n, nth = case["nz"], case["angles"]
    d1 = np.zeros(n)
    d1[0], d1[-1] = -1.0, 1.0
    kD = np.fft.fft(d1)
    kw, e1, e2 = (np.zeros((n, nth), complex) for _ in range(3))
    ed = np.zeros((n, nth))
    for l in range(nth):
        w = m["wav"][l].astype(np.float64)
        W, e3 = np.fft.fft(w), _diff3(w)
        n3, wn = math.sqrt((e3 * e3).sum()), float(m["wn"][l])
        if m["rt"] is None:
            kw[:, l], e1[:, l], e2[:, l] = W.conj() * kD, W.conj() / wn, np.fft.fft(e3).conj() / n3
            ed[:, l] = m["wnc"] * m["etc"][l, l]
        else:
            b = d1 - np.roll(d1, 1)
            kw[:, l], e1[:, l] = kD, 1.0 / wn
            e2[:, l] = np.fft.fft(0.5 * (np.roll(b, -1) - np.roll(b, 1))) / n3
            cn = n // 2 + 1
            k = np.arange(cn)
            om = k / 0.999
            lo = np.minimum(np.floor(om).astype(int), cn - 1)
            hi = np.minimum(lo + 1, cn - 1)
            v = np.where(om < cn, W[lo] * (1 - (om - lo)) + W[hi] * (om - lo), 0) / 0.999
            big = np.maximum(np.abs(W[:cn]) ** 2, np.abs(v) ** 2)
            r2 = np.where(big > 0, 1.0 / np.maximum(big, 1e-300), (wn * n * n * 100.0) ** 2)
            kk = np.minimum(np.arange(n), n - np.arange(n))
            ed[:, l] = m["wnc"] * m["etc"][l, l] * r2[kk]
    f = 1000.0 / (DT * n) * np.minimum(np.arange(n), n - np.arange(n))
    return kw, e1, e2, ed, (f > m["low"] * m["min_rt"]) & (f < m["high"])


def _prior_grids(case, m):
    """Spectra of the prior correlation and the error correlation with gradients, (nz, ny, cnx)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev = "cuda"
    cyc = lambda n: torch.where(torch.arange(n, device=dev) < n - torch.arange(n, device=dev),  # noqa: E731
                                torch.arange(n, device=dev), torch.arange(n, device=dev) - n).double()
    # the position subK is a float, rounded after each operation: at -1 the weight jumps
    at = (cyc(nx).float() * GRAD[0])[None, None, :], (cyc(ny).float() * GRAD[1])[None, :, None]
    sub = (torch.arange(nz, device=dev).float()[:, None, None] + at[0] + at[1]).double()
    cxy, ct = (torch.from_numpy(m[q].astype(np.float64)).cuda() for q in ("cxy", "cct"))
    base = torch.floor(sub)
    s = sub - base
    b0 = torch.remainder(base, nz).long()
    cov = ((1 - s) * ct[b0] + s * ct[(b0 + 1) % nz]) * cxy[None]
    # fillInErrCorr truncates towards zero: a subK in (-1, 0) weighs 1 - subK
    far = torch.clamp(1 - (sub - nz).abs(), min=0)
    err = torch.where(sub.abs() < 1, 1 - sub, far) * cxy[None]
    return torch.fft.rfftn(cov, dim=(0, 1, 2)).real.abs(), torch.fft.rfftn(err, dim=(0, 1, 2)).real.abs()


def _invert(case, seed):
    nx, ny, nz, nth, sims = case["nx"], case["ny"], case["nz"], case["angles"], case["sims"]
    dims = (nz, ny, nx)
    m = _model(case, seed)
    spec = []
    for l in range(nth + 3):
        g = torch.empty((nz, ny, 2 * (nx // 2 + 1)), device="cuda")
        _fill(g, nx, seed, l if l < nth else 16 + l - nth, None if l < nth else MEAN[l - nth])
        g = g[..., :nx].double()
        if l < nth and m["rt"] is not None:
            g = _divide(case, m, g, l)
        spec.append(torch.fft.rfftn(g, dim=(0, 1, 2), norm="ortho"))
        del g
    d, mu = spec[:nth], spec[nth:]
    kw, e1, e2, ed, inv = _kz(case, m)
    A, pv = m["A"], m["pv"]
    ec = 0.5 * (1.0 - m["wnc"]) * m["etc"]
    grids = case.get("prior") == "grids"
    if grids:
        R, E = _prior_grids(case, m)
    else:
        c2 = torch.fft.rfft2(torch.from_numpy(m["cxy"].astype(np.float64)).cuda())
        c1 = torch.from_numpy(np.fft.fft(m["cct"].astype(np.float64)).real).cuda()
    cov = [torch.empty((nz, ny, nx // 2 + 1), dtype=torch.complex128, device="cuda") for _ in range(6)]
    sim = [torch.empty((nz, ny, nx // 2 + 1), dtype=torch.complex128, device="cuda") for _ in range(3 * sims)]
    slab = max(1, 3_000_000 // (ny * (nx // 2 + 1)))
    G = A @ pv @ A.T
    AP = A @ pv
    for k0 in range(0, nz, slab):
        k1 = min(nz, k0 + slab)
        col = lambda v: torch.from_numpy(np.ascontiguousarray(v[k0:k1])).cuda()[:, None, None]  # noqa: E731
        if grids:
            rho, lam = R[k0:k1], E[k0:k1]
        else:
            rho = (c1[k0:k1, None, None] * c2.real[None]).abs()
            lam = c2.real.abs()[None].expand_as(rho)
        Sd = [[None] * nth for _ in range(nth)]
        for a in range(nth):
            for b in range(a + 1):
                kk = col(kw[:, a] * kw[:, b].conj())
                ee = col(e1[:, a] * e1[:, b].conj() + e2[:, a] * e2[:, b].conj())
                Sd[a][b] = rho * (G[a, b] * kk) + lam * (ec[a, b] * ee)
            Sd[a][a] = Sd[a][a] + col(ed[:, a])
        L, ok = _chol(Sd)
        del Sd
        ok = ok & torch.from_numpy(inv[k0:k1]).cuda()[:, None, None]
        KS = [[rho * (AP[l, a] * col(kw[:, l])) for l in range(nth)] for a in range(3)]
        X = [_solve(L, KS[a]) for a in range(3)]                     # Sd^-1 K S
        dm = [d[l][k0:k1] - col(kw[:, l]) * sum(A[l, a] * mu[a][k0:k1] for a in range(3)) for l in range(nth)]
        S = []
        for q, (a, b) in enumerate(PAIRS):
            red = sum(KS[a][l].conj() * X[b][l] for l in range(nth))
            S.append(rho * pv[a, b] - torch.where(ok, red, torch.zeros_like(red)))
            cov[q][k0:k1] = S[q]
        post = []
        for a in range(3):
            add = sum(X[a][l].conj() * dm[l] for l in range(nth))
            post.append(mu[a][k0:k1] + torch.where(ok, add, torch.zeros_like(add)))
        for l in range(nth):
            res = dm[l] - col(kw[:, l]) * sum(A[l, a] * (post[a] - mu[a][k0:k1]) for a in range(3))
            d[l][k0:k1] = torch.where(ok, res, d[l][k0:k1])
        for a in range(3):
            mu[a][k0:k1] = post[a]
        if sims:
            C = [[S[0]], [S[3].conj(), S[1]], [S[4].conj(), S[5].conj(), S[2]]]
            F, fine = _chol(C)
            for s in range(sims):
                z = _noise(int(seed), s, torch.arange(k0, k1, device="cuda"), ny, nz, nx)
                for a in range(3):
                    v = sum(F[a][b] * z[b] for b in range(a + 1))
                    sim[3 * s + a][k0:k1] = post[a] + torch.where(fine, v, torch.zeros_like(v))
    back = lambda g, norm: torch.fft.irfftn(g, s=dims, dim=(0, 1, 2), norm=norm)  # noqa: E731
    out = {"mean": torch.stack([back(g, "ortho") for g in mu]), "cov": torch.stack([back(g, "backward") for g in cov])}
    del cov
    if case.get("resid"):
        out["resid"] = torch.stack(d)
    if sims:
        out["sims"] = torch.empty((3 * sims,) + dims, dtype=torch.float64, device="cuda")
        for q in range(3 * sims):
            out["sims"][q] = back(sim[q], "ortho")
            sim[q] = None
    if case["op"] == "host" and sims:
        out["sims"] = out["sims"].reshape((sims, 3) + dims)
    return out


def exact(case, seed):
    """run()'s outputs for the same inputs, from torch and numpy in 64 bits."""
    seed = int(seed)
    op = case["op"]
    if op in ("run", "host"):
        return _invert(case, seed)
    if op == "batch":
        return [_invert(c, seed * 16 + i) for i, c in enumerate(_batch_cases(case))]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if op == "fft":
        g = torch.empty((nz, ny, 2 * (nx // 2 + 1)), device="cuda")
        _fill(g, nx, seed, 0)
        x = g[..., :nx].double()
        spec = torch.fft.rfftn(x, dim=(0, 1, 2), norm="backward" if case["covariance"] else "ortho")
        return {"spec": torch.view_as_real(spec).reshape(nz, ny, -1), "back": x}
    m = _facies_model(case, seed)
    nb, dv, vmin, Q = m["nb"], m["dv"], m["vmin"], m["sinv"]
    off = [(torch.where(torch.arange(n) <= n // 2, torch.arange(n), torch.arange(n) - n).double() * dv[d]).cuda()
           for d, n in enumerate(nb)]
    a, b, c = off[0][None, None, :], off[1][None, :, None], off[2][:, None, None]
    g = torch.exp(-0.5 * (a * a * Q[0, 0] + b * b * Q[1, 1] + c * c * Q[2, 2] + 2 * a * b * Q[1, 0] + 2 * a * c * Q[2, 0]
                          + 2 * b * c * Q[2, 1]))
    Fs = torch.fft.rfftn(g / g.sum())
    hist = torch.from_numpy(m["hist"].astype(np.float64)).cuda()
    dens = torch.stack([torch.fft.irfftn(torch.fft.rfftn(h) * Fs, s=h.shape, dim=(0, 1, 2)) for h in hist])
    post = _facies_mean(case, seed)[..., :nx].double()
    idx, wgt = [], []
    for q in range(3):
        f = (post[q] - vmin[q]) / dv[q] - 0.5
        i1 = torch.floor(f)
        edge = (i1 < 0) | (i1 >= nb[q] - 1)
        wgt.append(torch.where(edge, torch.zeros_like(f), f - i1))
        i1 = i1.long().clamp(0, nb[q] - 1)
        idx.append((i1, torch.where(edge, i1, (i1 + 1).clamp(max=nb[q] - 1))))
    undef = m["undef"] / float(nb[0] * nb[1] * nb[2])
    vals = []
    for f in range(case["facies"]):
        D = dens[f].clamp(min=0)
        v = 0.0
        for p in (0, 1):
            for q in (0, 1):
                for r in (0, 1):
                    w = (wgt[0] if p else 1 - wgt[0]) * (wgt[1] if q else 1 - wgt[1]) * (wgt[2] if r else 1 - wgt[2])
                    v = v + w * D[idx[2][r], idx[1][q], idx[0][p]]
        vals.append(float(m["prior"][f]) * v.clamp(min=0))
    s = undef + sum(vals)
    return {"dens": dens, "prob": torch.stack([v / s for v in vals] + [undef / s * torch.ones_like(s)])}
