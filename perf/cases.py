"""What a user has this framework do, as cases that can be timed and compared.

The framework samples the posterior of a Keplerian orbit by rejection: ln L of
prior samples against radial velocities of one or many stars, the acceptance
test, and the steps on either side (drawing the prior on the device, the
linear parameters of the accepted rows, radial-velocity curves).  Sizes are
those of the benchmark's configurations, of the tests and of ordinary use:
stars of 3 to 300 epochs over 1000 to 3000 days, periods of 2 to 1024 days,
from a hundred prior samples in one call to 2^27 in a device-resident cache.

A case's "kind" names the entry point (see the functions _prepare_*).
"""
import math

import numpy as np
import torch

from thejoker_gb300 import GPUJokerHelper, JokerPrior, JokerSamples, RVData, TheJoker
from thejoker_gb300 import device as dev
from thejoker_gb300.batch import BatchRejection
from thejoker_gb300.data import validate_prepare_data
from thejoker_gb300.iterative import IterativeBatch
from thejoker_gb300.pipeline import HostRejection
from thejoker_gb300.prior import LogNormal, Normal

P_MIN, P_MAX = 2.0, 1024.0
E_ALPHA, E_BETA = 0.867, 3.03
SIGMA_K0, P0, MAX_K = 30.0, 365.25, 500.0
SIGMA_V = (100.0, 1.0, 0.01)
SIGMA_OFFSET = 2.0
JITTER = (math.log(0.5), 1.0)
TWO_PI = 2.0 * math.pi
# sample-epochs that exact() evaluates in about ten seconds
EXACT_MOST = 100_000_000


def listed():
    return [
        # one small call of the drop-in helper on a host chunk, as a pool task
        # or a test makes it: three epochs, a hundred rows
        dict(name="lnl_call_small", kind="lnl", source="host", rows=97, epochs=3, poly=1,
             offsets=0, jitter=False),
        # the benchmark's small configuration: 16 epochs, 2^20 device samples
        dict(name="lnl_16_epochs", kind="lnl", source="device", rows=1 << 20, epochs=16, poly=1,
             offsets=0, jitter=False),
        # the default star (40 epochs, jitter applied) at the drop-in's precision
        dict(name="lnl_40_epochs_jitter", kind="lnl", source="device", rows=1_500_007, epochs=40,
             poly=1, offsets=0, jitter=True),
        # a long-observed star of two surveys with a quadratic trend: five
        # linear parameters, more epochs than one shared-memory tile
        dict(name="lnl_300_epochs_trend", kind="lnl", source="device", rows=60_013, epochs=300,
             poly=3, offsets=1, jitter=False),
        # the public call on a prior-sample table in memory, to posterior samples
        dict(name="rejection_call", kind="rejection", rows=131_071, epochs=21, poly=1,
             max_out=256),
        # a survey against one shared cache: stars of 3 to 256 epochs
        dict(name="batch_survey", kind="batch", stars=48, rows=400_009, epochs_min=3,
             epochs_max=256, poly=1, jitter=False, max_out=256),
        # the headline workload's star against a large cache
        dict(name="batch_one_star", kind="batch", stars=1, rows=1 << 27, epochs_min=40,
             epochs_max=40, poly=1, jitter=True, max_out=256),
        # adaptive rounds of many stars, quadratic trend
        dict(name="iterative_survey", kind="iterative", stars=96, rows=1 << 19, epochs_min=3,
             epochs_max=64, poly=3, requested=256),
        # a few stars against a chunk that lives in pinned host memory
        dict(name="host_chunk", kind="host", stars=4, rows=4_000_037, epochs_min=10,
             epochs_max=60, poly=1, jitter=False, max_out=256),
        # the linear parameters of many accepted rows, linear trend
        dict(name="posterior_rows", kind="posterior", rows=100_003, epochs=40, poly=2,
             jitter=False),
        # radial-velocity curves of posterior samples on a plotting grid
        dict(name="rv_curves", kind="rv", rows=4096, times=1001),
        # a prior cache drawn on the device, with the packed copy
        dict(name="prior_draw", kind="prior", rows=(1 << 24) + 77, jitter=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("lnl", "lnl", "lnl", "rejection", "batch", "batch", "iterative", "host",
                       "posterior", "rv", "prior"))
    c = dict(kind=kind)
    if kind == "lnl":
        c.update(source=rng.choice(("device", "device", "host")), epochs=_log_int(rng, 3, 300),
                 poly=rng.randint(1, 3), offsets=rng.choice((0, 0, 0, 1, 2)),
                 jitter=rng.random() < 0.4)
        c["rows"] = min(_log_int(rng, 1, 2_000_000), 60_000_000 // c["epochs"])
    elif kind == "rejection":
        c.update(rows=_log_int(rng, 1_000, 1_000_000), epochs=_log_int(rng, 3, 60),
                 poly=rng.randint(1, 2), max_out=rng.choice((128, 256, 512)))
    elif kind == "batch":
        c.update(stars=_log_int(rng, 1, 96), jitter=rng.random() < 0.5,
                 poly=rng.choice((1, 1, 2)), max_out=256)
        lo = _log_int(rng, 3, 64)
        c.update(epochs_min=lo, epochs_max=min(256, lo * rng.randint(1, 8)))
        c["rows"] = _log_int(rng, 4_096, 40_000_000 // c["stars"])
    elif kind == "iterative":
        c.update(stars=_log_int(rng, 1, 128), rows=_log_int(rng, 70_000, 1 << 19), epochs_min=3,
                 epochs_max=_log_int(rng, 16, 100), poly=rng.randint(1, 3),
                 requested=rng.choice((64, 128, 256)))
    elif kind == "host":
        c.update(stars=_log_int(rng, 1, 8), epochs_min=5, epochs_max=_log_int(rng, 16, 100),
                 poly=1, jitter=rng.random() < 0.5, max_out=256)
        c["rows"] = _log_int(rng, 10_000, 16_000_000 // c["stars"])
    elif kind == "posterior":
        c.update(rows=_log_int(rng, 16, 200_000), epochs=_log_int(rng, 3, 150),
                 poly=rng.randint(1, 3), jitter=rng.random() < 0.5)
    elif kind == "rv":
        c.update(rows=_log_int(rng, 1, 10_000), times=_log_int(rng, 7, 2_000))
    else:
        c.update(rows=_log_int(rng, 1_000, 1 << 24), jitter=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------ the inputs
def _eccentric_anomaly(x, e):
    """E of E - e sin E = x for x in [0, pi]: Halley's iteration from the
    upper end of the bracket [x, min(pi, x + e)], where the function is
    convex, in 32 bits first and then in 64."""
    def steps(x, e, E, n):
        for _ in range(n):
            s, c = torch.sin(E), torch.cos(E)
            f, f1, f2 = E - e * s - x, 1.0 - e * c, e * s
            E = E - 2.0 * f * f1 / torch.clamp(2.0 * f1 * f1 - f * f2, min=1e-30)
            E = torch.minimum(torch.maximum(E, x), x + e)
        return E
    xf, ef = x.float(), e.float()
    return steps(x, e, steps(xf, ef, torch.clamp(xf + ef, max=math.pi), 18).double(), 5)


def _unit_rv(dt, P, e, omega, M0):
    """cos(omega + f) + e cos(omega) at mean anomaly 2 pi dt / P - M0, 64 bits."""
    M = TWO_PI * (dt / P) - M0
    M = M - TWO_PI * torch.round(M / TWO_PI)
    E = torch.sign(M) * _eccentric_anomaly(M.abs(), e.expand_as(M))
    den = 1.0 - e * torch.cos(E)
    cos_f = (torch.cos(E) - e) / den
    sin_f = torch.sqrt((1.0 - e) * (1.0 + e)) * torch.sin(E) / den
    return torch.cos(omega) * (cos_f + e) - torch.sin(omega) * sin_f


def _chunk(rows, seed, jitter):
    """Packed prior samples (P, e, omega, M0, s) as the default prior draws
    them, a CUDA tensor."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = lambda: torch.rand(rows, dtype=torch.float64, device="cuda", generator=g)
    out = torch.empty((rows, 5), dtype=torch.float64, device="cuda")
    out[:, 0] = torch.exp(u() * math.log(P_MAX / P_MIN) + math.log(P_MIN))
    x, y = (torch._standard_gamma(torch.full((rows,), a, dtype=torch.float32, device="cuda"),
                                  generator=g).double() for a in (E_ALPHA, E_BETA))
    out[:, 1] = torch.clamp(x / (x + y), max=1.0 - 2.0 ** -24)
    out[:, 2] = u() * TWO_PI
    out[:, 3] = u() * TWO_PI
    if jitter:
        z = torch.randn(rows, dtype=torch.float64, device="cuda", generator=g)
        out[:, 4] = torch.exp(JITTER[0] + JITTER[1] * z)
    else:
        out[:, 4] = 0.0
    return out


def _star(rng, epochs, poly, offsets=0):
    """One star as a StarTable takes it (surveys one after the other in time),
    with its errors and the survey of each epoch."""
    base = rng.uniform(1000.0, 3000.0)
    t = 2456000.0 + np.sort(rng.uniform(0.0, base, epochs))
    err = rng.uniform(0.1, 1.0, epochs)
    survey = np.arange(epochs) * (offsets + 1) // epochs
    offsets = int(survey.max())
    dt = t - t[0]
    rv = rng.normal(0.0, 30.0) + rng.normal(0.0, err)
    if rng.uniform() < 0.6:
        P = math.exp(rng.uniform(math.log(P_MIN), math.log(P_MAX)))
        pars = [torch.tensor(v, dtype=torch.float64)
                for v in (P, rng.beta(E_ALPHA, E_BETA), *rng.uniform(0.0, TWO_PI, 2))]
        rv = rv + rng.uniform(1.0, 50.0) * _unit_rv(torch.from_numpy(dt), *pars).numpy()
    for j in range(1, poly):
        rv = rv + rng.normal(0.0, 0.1 * SIGMA_V[j]) * dt ** j
    for j in range(offsets):
        rv = rv + rng.normal(0.0, SIGMA_OFFSET) * (survey == j + 1)
    columns = [np.ones(epochs)] + [(survey == j + 1) * 1.0 for j in range(offsets)] + \
        [dt ** j for j in range(1, poly)]
    lam = [0.0, SIGMA_V[0] ** 2] + [SIGMA_OFFSET ** 2] * offsets + \
        [SIGMA_V[j] ** 2 for j in range(1, poly)]
    star = dict(t=t, rv=rv, ivar=1.0 / err ** 2, t_ref=t[0], trend_M=np.stack(columns, axis=1),
                mu=np.zeros(len(lam)), lam=np.array(lam),
                k_prior=np.array([1.0, SIGMA_K0, P0, MAX_K]))
    return star, err, survey


def _stars(case, seed):
    rng = np.random.default_rng(seed)
    lo, hi = math.log(case["epochs_min"]), math.log(case["epochs_max"])
    return [_star(rng, int(round(math.exp(rng.uniform(lo, hi)))), case["poly"])[0]
            for _ in range(case["stars"])]


def _one_star(case, seed):
    return _star(np.random.default_rng(seed), case["epochs"], case["poly"],
                 case.get("offsets", 0))


def _data_and_prior(case, seed):
    star, err, survey = _one_star(case, seed)
    n_off = int(survey.max())
    prior = JokerPrior.default(
        P_min=P_MIN, P_max=P_MAX, sigma_K0=SIGMA_K0, sigma_v=list(SIGMA_V[:case["poly"]]),
        poly_trend=case["poly"],
        v0_offsets=[(f"dv0_{j + 1}", Normal(0.0, SIGMA_OFFSET)) for j in range(n_off)])
    data = [RVData(star["t"][survey == j], star["rv"][survey == j], err[survey == j])
            for j in range(n_off + 1)]
    return data[0] if n_off == 0 else data, prior, n_off


def _jitter(case):
    return "applied" if case.get("jitter") else "reference"


def _seeds(case, seed):
    return [seed * 1000 + k for k in range(case["stars"])]


# ------------------------------------------------------- the entry points' states
def _prepare_lnl(case, seed):
    data, prior, n_off = _data_and_prior(case, seed)
    all_data, _, trend = validate_prepare_data(data, case["poly"], n_off)
    helper = GPUJokerHelper(all_data, prior, trend, precision="fp64", jitter=_jitter(case))
    chunk = _chunk(case["rows"], seed, case["jitter"])
    return dict(helper=helper, chunk=chunk if case["source"] == "device" else chunk.cpu().numpy())


def _prepare_rejection(case, seed):
    data, prior, _ = _data_and_prior(case, seed)
    cols = _chunk(case["rows"], seed, False).cpu().numpy()
    table = JokerSamples({k: cols[:, i] for i, k in enumerate(("P", "e", "omega", "M0", "s"))})
    return dict(data=data, prior=prior, table=table, seed=seed)


def _prepare_batch(case, seed):
    cache = dev.PriorCache.from_samples(_chunk(case["rows"], seed, case["jitter"]))
    return dict(batch=BatchRejection(_stars(case, seed), cache, jitter=_jitter(case),
                                     max_out=case["max_out"], seeds=_seeds(case, seed)))


def _prepare_iterative(case, seed):
    cache = dev.PriorCache.from_samples(_chunk(case["rows"], seed, False))
    seeds = _seeds(case, seed)
    engine = IterativeBatch(dev.StarTable(_stars(case, seed)), cache, case["requested"],
                            seeds=seeds)
    return dict(engine=engine, seeds=seeds)


def _prepare_host(case, seed):
    table = dev.StarTable(_stars(case, seed), jitter=_jitter(case))
    chunk = _chunk(case["rows"], seed, case["jitter"]).cpu().pin_memory()
    states = [dev.pcg64_state(np.random.default_rng(s)) for s in _seeds(case, seed)]
    return dict(engine=HostRejection(table, case["rows"], max_out=case["max_out"]), chunk=chunk,
                states=states)


def _prepare_posterior(case, seed):
    table = dev.StarTable([_one_star(case, seed)[0]], jitter=_jitter(case))
    cache = dev.PriorCache.from_samples(_chunk(case["rows"], seed, case["jitter"]))
    rows = torch.randperm(case["rows"], generator=torch.Generator().manual_seed(seed))
    return dict(table=table, cache=cache, rows=rows.cuda())


def _curves(case, seed):
    c = _chunk(case["rows"], seed, False)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    K = 5.0 + 45.0 * torch.rand(case["rows"], dtype=torch.float64, device="cuda", generator=g)
    start = 2456000.0 + 10.0 * (seed % 97)
    t = torch.linspace(start, start + 2000.0, case["times"], dtype=torch.float64, device="cuda")
    return torch.stack([c[:, 0], K, c[:, 1], c[:, 2], c[:, 3]], dim=1).contiguous(), t, start


def _prepare_rv(case, seed):
    elems, t, t0 = _curves(case, seed)
    return dict(elems=elems, t=t, t0=t0)


def _prepare_prior(case, seed):
    prior = JokerPrior.default(P_min=P_MIN, P_max=P_MAX, sigma_K0=SIGMA_K0, sigma_v=SIGMA_V[0],
                               s=LogNormal(*JITTER) if case["jitter"] else None)
    packed = torch.empty((case["rows"], 5), dtype=torch.float64, device="cuda")
    return dict(prior=prior, cache=dev.PriorCache(case["rows"]), packed=packed, seed=seed)


_PREPARE = dict(lnl=_prepare_lnl, rejection=_prepare_rejection, batch=_prepare_batch,
                iterative=_prepare_iterative, host=_prepare_host, posterior=_prepare_posterior,
                rv=_prepare_rv, prior=_prepare_prior)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    state["source"] = case.get("source")
    state["max_out"] = case.get("max_out", case.get("requested"))
    return state


# --------------------------------------------------------------------- one pass
def _padded(rows, width, fill):
    """Ragged rows (what was kept, star by star) as one array of fixed width."""
    out = np.full((len(rows), width), fill)
    for k, r in enumerate(rows):
        out[k, :len(r)] = r
    return out


def run(state):
    kind = state["kind"]
    if kind == "lnl":
        if state["source"] == "host":
            return state["helper"].batch_marginal_ln_likelihood(state["chunk"])
        return state["helper"].batch_marginal_ln_likelihood_device(state["chunk"])
    if kind == "rejection":
        joker = TheJoker(state["prior"], rng=np.random.default_rng(state["seed"]))
        out = joker.rejection_sample(state["data"], state["table"],
                                     max_posterior_samples=state["max_out"], in_memory=True)
        return {k: _padded([out[k]], state["max_out"], 0.0) for k in out.keys()}
    if kind == "batch":
        counts, idx, lnl = state["batch"].run().results()
        return dict(counts=counts, idx=_padded(idx, state["max_out"], -1),
                    lnl=_padded(lnl, state["max_out"], 0.0))
    if kind == "iterative":
        rows, idx, _ = state["engine"].reset(state["seeds"]).run().results()
        return dict(state=rows, idx=_padded(idx, state["max_out"], -1))
    if kind == "host":
        counts, idx = state["engine"].run(state["chunk"], state["states"])
        return dict(counts=counts, idx=_padded(idx, state["max_out"], -1))
    if kind == "posterior":
        a, A, lnl = dev.linear_posterior(state["table"], state["cache"], 0, state["rows"])
        return dict(a=a, A=A, lnl=lnl)
    if kind == "rv":
        return dev.rv_from_elements(state["t"], state["elems"], state["t0"])
    state["cache"].sample_prior(state["prior"], seed=state["seed"], packed=state["packed"])
    P, e, omega, M0, s = state["packed"].unbind(1)
    return dict(P=P, e=e, omega=omega, M0=M0, s=s)


# ------------------------------------------------------------------------- work
# flops of one (sample, epoch) and of one sample's solve, as the benchmark
# counts them (a Kepler solve, the velocity column and the epoch sums)
_EPOCH_FLOPS, _SAMPLE_FLOPS = 62, 21


def work(case):
    kind, rows = case["kind"], case["rows"]
    if kind in ("lnl", "rejection"):
        flops = rows * (case["epochs"] * _EPOCH_FLOPS + _SAMPLE_FLOPS)
        return dict(bytes=rows * 48, flops=flops)
    if kind in ("batch", "iterative", "host"):
        lo, hi = case["epochs_min"], case["epochs_max"]
        mean = lo if hi == lo else (hi - lo) / math.log(hi / lo)
        # adaptive rounds evaluate at least their first batch
        each = 128 * case["requested"] if kind == "iterative" else rows
        return dict(bytes=rows * 40,
                    flops=case["stars"] * each * (mean * _EPOCH_FLOPS + _SAMPLE_FLOPS))
    if kind == "posterior":
        L = 1 + case["poly"]
        return dict(bytes=rows * (48 + 8 * (L + L * L + 1)),
                    flops=rows * (case["epochs"] * (_EPOCH_FLOPS + L * (L + 3)) + L ** 3))
    if kind == "rv":
        return dict(bytes=rows * 40 + 8 * case["times"] * (1 + rows),
                    flops=rows * case["times"] * _EPOCH_FLOPS)
    # the packed rows and the cache's two forms of them
    return dict(bytes=rows * (40 + 76), flops=rows * 200)


# ------------------------------------------------------------------ exact values
def _blocks(n, epochs):
    step = max(1, 40_000_000 // epochs)
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _system(star, chunk, jitter, clip):
    """G, q, Lambda_0, r^T W r and sum log w of rows of prior samples."""
    put = lambda v: torch.as_tensor(v, dtype=torch.float64, device=chunk.device)
    P, e, omega, M0, s = (chunk[:, k:k + 1] for k in range(5))
    m = _unit_rv(put(star["t"] - star["t_ref"])[None, :], P, e, omega, M0)
    ivar, y, T = put(star["ivar"])[None, :], put(star["rv"])[None, :], put(star["trend_M"])
    w = ivar / (1.0 + s * s * ivar) if jitter else ivar.expand_as(m)
    lam0 = SIGMA_K0 ** 2 / (1.0 - e[:, 0] ** 2) * (P[:, 0] / P0) ** (-2.0 / 3.0)
    if clip:
        lam0 = torch.clamp(lam0, max=MAX_K ** 2)
    L = 1 + T.shape[1]
    G = torch.empty((len(chunk), L, L), dtype=torch.float64, device=chunk.device)
    q = torch.empty((len(chunk), L), dtype=torch.float64, device=chunk.device)
    cols = [m] + [T[:, j][None, :].expand_as(m) for j in range(L - 1)]
    for i in range(L):
        wc = w * cols[i]
        q[:, i] = (wc * y).sum(1)
        for k in range(i + 1):
            G[:, i, k] = G[:, k, i] = (wc * cols[k]).sum(1)
        G[:, i, i] += 1.0 / (lam0 if i == 0 else star["lam"][i])
    return G, q, lam0, (w * y * y).sum(1), torch.log(w).sum(1)


def _ln_likelihood(star, chunk, jitter, clip=True):
    """ln L, and the mean and covariance of the linear parameters."""
    G, q, lam0, yy, logw = _system(star, chunk, jitter, clip)
    d = torch.rsqrt(torch.diagonal(G, dim1=1, dim2=2))            # scaled to a unit diagonal
    C = torch.linalg.cholesky(G * d[:, :, None] * d[:, None, :])
    z = torch.linalg.solve_triangular(C, (q * d)[:, :, None], upper=False)[:, :, 0]
    logdet = 2.0 * (torch.log(torch.diagonal(C, dim1=1, dim2=2)) - torch.log(d)).sum(1)
    logdet = logdet + torch.log(lam0) + float(np.log(star["lam"][1:]).sum()) - logw + \
        len(star["t"]) * math.log(TWO_PI)
    A = torch.cholesky_inverse(C) * d[:, :, None] * d[:, None, :]
    return -0.5 * (yy - (z * z).sum(1) + logdet), torch.einsum("nij,nj->ni", A, q), A


def _all_ln_likelihoods(star, chunk, jitter):
    return torch.cat([_ln_likelihood(star, chunk[a:b], jitter)[0]
                      for a, b in _blocks(len(chunk), len(star["t"]))])


def _accepted(lnl, u, max_out):
    d = (lnl - lnl.max()).cpu().numpy()
    good = np.where(np.exp(d) > u)[0]
    return len(good), good[:max_out]


def _philox(counter, key):
    """Philox4x32-10 on int64 tensors that hold 32-bit words."""
    low = 0xFFFFFFFF
    c, k = list(counter), list(key)
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        h0, h1 = (p0 >> 32) & low, (p1 >> 32) & low
        c = [h1 ^ c[1] ^ k[0], p1 & low, h0 ^ c[3] ^ k[1], p0 & low]
        k = [(k[0] + 0x9E3779B9) & low, (k[1] + 0xBB67AE85) & low]
    return c


def _exact_prior(case, seed):
    """P, omega and M0 from the counter-based stream of each sample (e and s
    are random draws of a rejection sampler in 32 bits)."""
    g = torch.arange(case["rows"], dtype=torch.int64, device="cuda")
    zero = torch.zeros_like(g)
    u = []
    for block in (0, 1):
        w = _philox((g, zero, zero + block, zero + 0x4A6F6B72), (seed, 0))
        u += [((w[2 * h + 1] << 21) | (w[2 * h] >> 11)).double() * 2.0 ** -53 for h in (0, 1)]
    span = math.log(P_MAX) - math.log(P_MIN)
    return dict(P=torch.exp(u[0] * span + math.log(P_MIN)), e=None, omega=u[1] * TWO_PI,
                M0=u[2] * TWO_PI, s=None)


def exact(case, seed):
    kind = case["kind"]
    if kind == "lnl":
        chunk = _chunk(case["rows"], seed, case["jitter"])
        return _all_ln_likelihoods(_one_star(case, seed)[0], chunk, case["jitter"])
    if kind == "rejection":
        star = _one_star(case, seed)[0]
        chunk = _chunk(case["rows"], seed, False)
        rng = np.random.default_rng(seed)
        lnl = _all_ln_likelihoods(star, chunk, False)
        _, good = _accepted(lnl, rng.uniform(size=len(lnl)), case["max_out"])
        kept = chunk[torch.from_numpy(good).cuda()]
        _, a, A = _ln_likelihood(star, kept, False, clip=False)
        rows = np.array([rng.multivariate_normal(m, C) for m, C in zip(a.cpu().numpy(),
                                                                       A.cpu().numpy())])
        out = dict(zip(("P", "e", "omega", "M0", "s"), kept.cpu().numpy().T))
        out.update(zip(["K"] + [f"v{j}" for j in range(case["poly"])], rows.T))
        return {k: _padded([v], case["max_out"], 0.0) for k, v in out.items()}
    if kind == "batch":
        stars = _stars(case, seed)
        if case["rows"] * sum(len(s["t"]) for s in stars) > EXACT_MOST:
            return None
        chunk, out = _chunk(case["rows"], seed, case["jitter"]), dict(counts=[], idx=[], lnl=[])
        for star, sd in zip(stars, _seeds(case, seed)):
            lnl = _all_ln_likelihoods(star, chunk, case["jitter"])
            n, good = _accepted(lnl, np.random.default_rng(sd).uniform(size=len(lnl)),
                                case["max_out"])
            out["counts"].append(n)
            out["idx"].append(good)
            out["lnl"].append(lnl.cpu().numpy()[good])
        return dict(counts=np.array(out["counts"]), idx=_padded(out["idx"], case["max_out"], -1),
                    lnl=_padded(out["lnl"], case["max_out"], 0.0))
    if kind == "posterior":
        star = _one_star(case, seed)[0]
        chunk = _chunk(case["rows"], seed, case["jitter"])
        rows = torch.randperm(case["rows"], generator=torch.Generator().manual_seed(seed)).cuda()
        parts = [_ln_likelihood(star, chunk[rows[a:b]], case["jitter"], clip=False)
                 for a, b in _blocks(case["rows"], case["epochs"])]
        lnl, a, A = (torch.cat(p) for p in zip(*parts))
        return dict(a=a, A=A, lnl=lnl)
    if kind == "rv":
        elems, t, t0 = _curves(case, seed)
        P, K, e, omega, M0 = (elems[:, k:k + 1] for k in range(5))
        return torch.cat([K[a:b] * _unit_rv((t - t0)[None, :], P[a:b], e[a:b], omega[a:b],
                                            M0[a:b]) for a, b in _blocks(len(elems), len(t))])
    if kind == "prior":
        return _exact_prior(case, seed)
    return None
