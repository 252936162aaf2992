"""Performance cases of the slip-link simulator: what a user of the package has it do.

Every case is one pass of a program that keeps its ensembles resident: the next
window of an equilibrium melt with its correlator, of a flow, of a batch or a
polydisperse melt, the next output series, a window from conformations in host
memory, the statistics files of a state, or a batch of served requests.

listed()             the cases by name
draw(rng)            one more case of the same ranges
prepare(case, seed)  the ensembles (or server, or device buffers) a program keeps
run(state)           one pass through the public entry points
work(case)           bytes and operations a pass cannot do without
exact(case, seed)    64-bit results, where they do not depend on a trajectory
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import gpu_dsm_gb300 as dsm

P_END = 1.0e7  # run length (tau_K) that sizes the correlators, as in a production run


def listed():
    return [
        # the smallest call: the 1024-chain, N_K = 25 melt with G(t), advanced one
        # sample interval; launches and host work count here
        dict(name="melt_nk25_1tau", kind="melt", mode="gt", n=1024, nk=25, beta=1.0, p=16, m=2, window=1.0),
        # a served G(t) request of ordinary size, more activity, short correlator
        dict(name="melt_nk50_beta2", kind="melt", mode="gt", n=16384, nk=50, beta=2.0, p=16, m=2, window=50.0),
        # the headline melt: 65536 chains of N_K = 200 with G(t)
        dict(name="melt_nk200", kind="melt", mode="gt", n=65536, nk=200, beta=1.0, p=64, m=8, window=150.0),
        # long, strongly entangled chains (odd N_K, beta = 0.5: Z near 309)
        dict(name="melt_nk463_long", kind="melt", mode="gt", n=4096, nk=463, beta=0.5, p=64, m=8, window=50.0),
        # centre-of-mass diffusion (eq_type 2)
        dict(name="msd_nk100", kind="melt", mode="msd", n=8192, nk=100, beta=1.0, p=64, m=8, window=50.0),
        # polydisperse melt, log-normal N_K, PDI 1.5
        dict(name="poly_lognormal", kind="poly", n=32768, mean=150, pdi=1.5, most=1000, window=40.0),
        # shear start-up at four rates in one batched launch
        dict(name="shear_batch_nk100", kind="shear", n=16384, nk=100, beta=1.0, wi_low=0.1, wi_high=100.0, rates=4,
             window=25.0),
        # a tau.dat series: 20 stress outputs of one small ensemble, elongation
        dict(name="series_nk50", kind="series", n=4096, nk=50, beta=1.0, flow="elongation", wi=10.0, dt=2.5, outputs=20),
        # caller-owned device buffers, no correlator, odd N_K
        dict(name="buffers_nk131", kind="buffers", n=32768, nk=131, beta=1.0, wi=0.0, window=25.0),
        # conformations from host memory, a window, conformations and G(t) back
        dict(name="restart_nk75", kind="restart", n=16384, nk=75, beta=1.0, p=64, m=8, window=25.0),
        # the -distr statistics and the stress of a state handed in by the user
        dict(name="stats_nk150", kind="stats", n=32768, nk=150, beta=1.0),
        # served requests: half G(t), half shear, short runs
        dict(name="serve_8", kind="serve", requests=8, nk_low=20, nk_high=300, n_low=1024, n_high=8192, t_end=40.0),
    ]


def draw(rng):
    lu = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    # a pass of at most this many chain-tau_K x N_K: below the largest listed case
    most = 65536 * 200 * 150.0
    kind = rng.choice(["melt", "melt", "melt", "poly", "shear", "series", "buffers", "restart", "stats", "serve"])
    nk = int(round(lu(20, 500)))
    n = int(round(lu(1024, 65536)))
    n = max(1024, min(n, int(8.0e6 / nk)))  # conformations of at most 160 MB
    beta = rng.choice([0.5, 1.0, 2.0])
    window = round(min(lu(1.0, 150.0), 0.2 * most / (n * nk)), 2)
    if kind == "melt":
        p, m = rng.choice([(16, 2), (64, 8), (32, 4)])
        return dict(kind="melt", mode=rng.choice(["gt", "gt", "msd", "none"]), n=n, nk=nk, beta=beta, p=p, m=m,
                    window=window)
    if kind == "poly":
        return dict(kind="poly", n=int(lu(4096, 32768)), mean=int(lu(40, 150)), pdi=rng.choice([1.1, 1.5, 2.0]),
                    most=int(lu(400, 1000)), window=round(lu(2.0, 40.0), 1))
    if kind == "shear":
        return dict(kind="shear", n=int(lu(1024, 16384)), nk=int(lu(20, 200)), beta=beta, wi_low=0.1,
                    wi_high=rng.choice([10.0, 100.0]), rates=rng.randint(2, 4), window=round(lu(2.0, 20.0), 1))
    if kind == "series":
        return dict(kind="series", n=int(lu(512, 8192)), nk=int(lu(20, 200)), beta=beta,
                    flow=rng.choice(["shear", "elongation"]), wi=round(lu(0.1, 50.0), 3), dt=round(lu(0.5, 5.0), 2),
                    outputs=rng.randint(3, 40))
    if kind == "buffers":
        return dict(kind="buffers", n=min(n, 32768), nk=int(lu(20, 300)), beta=beta, wi=rng.choice([0.0, 0.0, 5.0]),
                    window=round(lu(1.0, 20.0), 1))
    if kind == "restart":
        return dict(kind="restart", n=min(n, 32768), nk=int(lu(20, 200)), beta=beta, p=64, m=8,
                    window=round(lu(1.0, 25.0), 1))
    if kind == "stats":
        return dict(kind="stats", n=min(n, 32768), nk=int(lu(20, 200)), beta=beta)
    return dict(kind="serve", requests=rng.randint(3, 12), nk_low=20, nk_high=int(lu(60, 300)), n_low=1024,
                n_high=int(lu(2048, 8192)), t_end=round(lu(5.0, 40.0), 1))


# ------------------------------------------------------------------ helpers
def _kappa(flow, rate):
    if flow == "elongation":
        return (rate, 0.0, 0.0, 0.0, -0.5 * rate, 0.0, 0.0, 0.0, -0.5 * rate)
    return (0.0, rate, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0)


def _wis(case):
    k = case["rates"]
    return [case["wi_low"] * (case["wi_high"] / case["wi_low"]) ** (i / (k - 1)) for i in range(k)]


def _poly_nk(case, seed):
    rng = np.random.default_rng(seed)
    s2 = math.log(case["pdi"])
    v = np.exp(rng.normal(math.log(case["mean"]) - s2 / 2, math.sqrt(s2), size=case["n"]))
    return np.clip(np.round(v), 10, case["most"]).astype(np.int32)


def _requests(case, seed):
    """A request stream as the serving benchmark draws it: half G(t), half steady shear."""
    rng = np.random.default_rng(seed)
    lu = lambda a, b: float(np.exp(rng.uniform(math.log(a), math.log(b))))  # noqa: E731
    out = []
    for i in range(case["requests"]):
        nk = int(round(lu(case["nk_low"], case["nk_high"])))
        beta = float(rng.choice([0.5, 1.0, 2.0]))
        r = dict(nk=nk, beta=beta, n_chains=int(round(lu(case["n_low"], case["n_high"]))),
                 t_end=case["t_end"], seed=int(rng.integers(1, 1 << 31)), stream=i)
        if i % 2:
            r.update(kappa=_kappa("shear", lu(0.1, 100.0) / dsm.pcd(beta, nk)["tau_d"]), sync_dt=r["t_end"] / 10.0)
        else:
            r.update(eq_type=1, sync_dt=1.0, corr_p=16, corr_m=2)
        out.append(r)
    return out


def _host(n, cap):
    """Pinned host arrays in the reference layout, with their numpy views."""
    t = (torch.zeros(n * 16, dtype=torch.uint8, pin_memory=True), torch.zeros(n * cap * 4, pin_memory=True),
         torch.zeros(n * cap, pin_memory=True))
    return (t[0].numpy().view(dsm.HEAD_DTYPE), t[1].numpy().reshape(n, cap, 4), t[2].numpy().reshape(n, cap)), t


def _strands(case, seed):
    """Equilibrium conformations made with numpy: heads, {Q, N} and lifetime rates.
    Every seed gives the same strand sizes to other chains and other vectors and
    rates to all strands, so that the lists of strands have one length."""
    n, nk = case["n"], case["nk"]
    rng = np.random.default_rng(seed)
    cut = np.random.default_rng(n + nk).random((n, nk), dtype=np.float32) < 1.0 / (1.0 + case["beta"])
    cut[:, -1] = True  # the last Kuhn step ends the last strand
    cut = cut[rng.permutation(n)]
    c, k = np.nonzero(cut)
    Z = cut.sum(axis=1).astype(np.int32)
    start = np.concatenate([[0], np.cumsum(Z)[:-1]])
    i = np.arange(len(c)) - start[c]
    before = np.concatenate([[-1], k[:-1]])
    before[i == 0] = -1
    N = (k - before).astype(np.float32)
    q = rng.standard_normal((len(c), 3), dtype=np.float32) * np.sqrt(N / 3.0)[:, None].astype(np.float32)
    q[(i == 0) | (i == Z[c] - 1)] = 0.0  # the ends dangle
    heads = np.zeros(n, dsm.HEAD_DTYPE)
    heads["Z"] = Z
    qn = np.zeros((n, nk, 4), np.float32)
    qn[c, i, :3] = q
    qn[c, i, 3] = N
    tau = np.zeros((n, nk), np.float32)
    inner = i < Z[c] - 1
    tau[c[inner], i[inner]] = (10.0 ** rng.uniform(-4.0, 0.0, int(inner.sum()))).astype(np.float32)
    return heads, qn, tau


def _chains(ens, host):
    """The whole state of an ensemble, read back as a program that saves it does."""
    heads, qn, tau = ens.get_chains(out=host)
    ext = ens.get_ext()
    return {"Z": heads["Z"], "qn": qn, "tau": tau, "T": ext["T"], "step": ext["step"].view(np.int64),
            "dt": ext["dt_prev"], "stall": ext["stall"], "S": ext["S"], "hash": ext["hash"].view(np.int64)}


# ------------------------------------------------------------------ what a program keeps
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "t": 0.0}
    if kind in ("melt", "poly"):
        kw = dict(sync_dt=1.0, t_end=P_END, seed=seed, n_chains=case["n"])
        if kind == "poly":
            nkc = _poly_nk(case, seed)
            kw.update(nk=int(nkc.max()), nk_chain=nkc, eq_type=1, corr_p=64, corr_m=8)
        else:
            kw.update(nk=case["nk"], beta=case["beta"], eq_type={"gt": 1, "msd": 2, "none": 0}[case["mode"]],
                      corr_p=case["p"], corr_m=case["m"])
        s["ens"] = dsm.Ensemble(**kw)
        s["ens"].init_equilibrium()
    elif kind == "shear":
        tau_d = dsm.pcd(case["beta"], case["nk"])["tau_d"]
        s["ens"] = [dsm.Ensemble(nk=case["nk"], n_chains=case["n"], beta=case["beta"], kappa=_kappa("shear", w / tau_d),
                                 sync_dt=case["window"], t_end=P_END, seed=seed, stream=k)
                    for k, w in enumerate(_wis(case))]
        for e in s["ens"]:
            e.init_equilibrium()
    elif kind == "series":
        rate = case["wi"] / dsm.pcd(case["beta"], case["nk"])["tau_d"]
        s["ens"] = dsm.Ensemble(nk=case["nk"], n_chains=case["n"], beta=case["beta"], kappa=_kappa(case["flow"], rate),
                                sync_dt=case["dt"], t_end=P_END, seed=seed)
        s["ens"].init_equilibrium()
    elif kind == "buffers":
        n, nk = case["n"], case["nk"]
        rate = case["wi"] / dsm.pcd(case["beta"], nk)["tau_d"]
        e = dsm.Ensemble(nk=nk, n_chains=n, beta=case["beta"], kappa=_kappa("shear", rate), seed=seed)
        e.init_equilibrium()
        heads, qn, tau = e.get_chains()
        ext = e.get_ext()
        st = np.zeros(n, np.dtype([("Z", np.int32), ("stall", np.int32), ("S", np.int32), ("dt", np.float32),
                                   ("T", np.int64), ("step", np.uint64), ("hash", np.uint64), ("k", np.int64),
                                   ("nk", np.int32), ("pad", np.int32, 3)]))
        st["Z"], st["S"], st["hash"], st["nk"] = heads["Z"], ext["S"], ext["hash"], nk
        s.update(params=e.params, qn=torch.from_numpy(qn).cuda(), tau=torch.from_numpy(tau).cuda(),
                 st=torch.from_numpy(st.view(np.uint8)).cuda(), stress=torch.zeros(n * 8, device="cuda"))
        e.close()
        s["lib"] = lib = dsm.load_library()
        lib.dsm_advance_noalloc.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_double,
                                            C.c_int64, C.c_void_p, C.c_void_p]
        lib.dsm_advance_noalloc.restype = C.c_int
    elif kind in ("restart", "stats"):
        heads, qn, tau = _strands(case, seed)
        host, keep = _host(case["n"], case["nk"])
        host[0][:], host[1][:], host[2][:] = heads, qn, tau
        kw = {} if kind == "stats" else dict(eq_type=1, sync_dt=1.0, t_end=P_END, corr_p=case["p"], corr_m=case["m"])
        s["ens"] = dsm.Ensemble(nk=case["nk"], n_chains=case["n"], beta=case["beta"], seed=seed, **kw)
        s.update(given=host, given_keep=keep)
        if kind == "stats":
            s["ens"].set_chains(*host)
    else:
        s["requests"] = _requests(case, seed)
        s["server"] = dsm.Server(chunk_s=0.05)
    if kind in ("melt", "poly", "series", "restart"):
        s["host"], s["keep"] = _host(case["n"], s["ens"].z_max)
    if kind == "shear":
        s["host"] = [_host(case["n"], case["nk"]) for _ in s["ens"]]
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("melt", "poly"):
        s["t"] += case["window"]
        out = {"events": s["ens"].advance(s["t"]), **_chains(s["ens"], s["host"])}
        if kind == "poly" or case["mode"] != "none":
            out["gsum"], out["gcount"] = s["ens"].gt_raw()
        if kind == "melt" and case["mode"] == "msd":
            out["r1"] = s["ens"].r1()
        return out
    if kind == "shear":
        s["t"] += case["window"]
        ev = dsm.advance_batch(s["ens"], s["t"])
        return {"events": ev.view(np.int64), "stress": [e.stress()[0] for e in s["ens"]],
                "chains": [_chains(e, h[0]) for e, h in zip(s["ens"], s["host"])]}
    if kind == "series":
        ev, stress = s["ens"].advance_series(case["dt"], case["outputs"])
        return {"events": ev, "stress": stress, **_chains(s["ens"], s["host"])}
    if kind == "buffers":
        s["t"] += case["window"]
        ptr = [C.c_void_p(s[k].data_ptr()) for k in ("qn", "tau", "st", "stress")]
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = s["lib"].dsm_advance_noalloc(C.byref(s["params"]), *ptr, s["t"], -1, stream, None)
        if rc != 0:
            raise RuntimeError("dsm_advance_noalloc: %d" % rc)
        return {"qn": s["qn"], "tau": s["tau"], "state": s["st"], "stress": s["stress"]}
    if kind == "restart":
        s["ens"].set_chains(*s["given"])
        ev = s["ens"].advance(case["window"])
        out = {"events": ev, **_chains(s["ens"], s["host"])}
        out["gsum"], out["gcount"] = s["ens"].gt_raw()
        return out
    if kind == "stats":
        stress, count = s["ens"].stress()
        hz, hn, q = s["ens"].distributions()
        return {"stress": stress, "count": count, "hz": hz.view(np.int64), "hn": hn.view(np.int64), "q": q}
    srv = s["server"]
    ids = [srv.submit(**r) for r in s["requests"]]
    srv.wait_all(600.0)
    out = {"events": np.array([srv.status(i)["events"] for i in ids], np.int64)}
    for k, (i, r) in enumerate(zip(ids, s["requests"])):
        out["r%02d" % k] = srv.result_gt(i) if r.get("eq_type") == 1 else srv.result_stress(i)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _events(n, nk, tau):
    """kMC events of n chains over tau: the total rate of a chain is near 0.21 N_K + 0.5 per tau_K."""
    return n * tau * (0.21 * nk + 0.5)


def _melt_flops(events, samples, z, p):
    # per event six sliding rates (about 30 operations each), dt, pick and the
    # strand update; per sample the stress over strands and p lags
    return events * 240.0 + samples * (7.0 * z + 8.0 * p)


def _flow_flops(events, z):
    # per event every strand is deformed (24) and every pair's two sliding rates recomputed
    return events * (24.0 * z + 62.0 * (z - 1.0) + 60.0)


def _chain_bytes(n, z):
    return n * (20.0 * z + 64.0)


def work(case):
    kind = case["kind"]
    if kind == "serve":
        b = f = 0.0
        for r in _requests(case, 1):
            z = 1.0 + (r["nk"] - 1) / (1.0 + r["beta"])
            ev = _events(r["n_chains"], r["nk"], r["t_end"])
            f += _flow_flops(ev, z) if "kappa" in r else _melt_flops(ev, r["n_chains"] * r["t_end"], z, 16)
            b += 2.0 * _chain_bytes(r["n_chains"], z)
        return {"bytes": b, "flops": f}
    n, beta = case["n"], case.get("beta", 1.0)
    nk = case["mean"] if kind == "poly" else case["nk"]
    z = 1.0 + (nk - 1) / (1.0 + beta)
    if kind == "stats":
        return {"bytes": 2.0 * n * 16.0 * z, "flops": n * z * 40.0}
    # the chains in and out once, and the whole state handed to the caller
    b = 3.0 * _chain_bytes(n, z)
    if kind == "shear":
        return {"bytes": case["rates"] * b, "flops": case["rates"] * _flow_flops(_events(n, nk, case["window"]), z)}
    if kind == "series":
        return {"bytes": b, "flops": _flow_flops(_events(n, nk, case["dt"] * case["outputs"]), z)}
    ev = _events(n, nk, case["window"])
    if kind == "buffers":
        return {"bytes": 2.0 * _chain_bytes(n, z),
                "flops": _flow_flops(ev, z) if case["wi"] else _melt_flops(ev, 0.0, z, 0)}
    p, corr = case.get("p", 64), case.get("mode") != "none"
    if corr:
        b += 2.0 * n * 20.0 * p  # level 0 of the correlator in and out
    if kind == "restart":
        b += _chain_bytes(n, z)
    return {"bytes": b, "flops": _melt_flops(ev, n * case["window"] if corr else 0.0, z, p)}


def exact(case, seed):
    """The statistics of a given state in 64 bits.  The other cases follow a
    random trajectory whose every step depends on the last one's rounding."""
    if case["kind"] != "stats":
        return None
    heads, qn, _ = _strands(case, seed)
    q, N, Z = qn[:, :, :3].astype(np.float64), qn[:, :, 3].astype(np.float64), heads["Z"].astype(np.int64)
    w = np.where(N > 0, 3.0 / np.where(N > 0, N, 1.0), 0.0)
    pair = lambda a, b: -(q[:, :, a] * q[:, :, b] * w).sum(axis=1).mean()  # noqa: E731
    ln = np.sqrt((q * q).sum(axis=2))
    stress = [pair(0, 0), pair(1, 1), pair(2, 2), pair(0, 1), pair(1, 2), pair(0, 2), ln.sum(axis=1).mean(), Z.mean()]
    cap = case["nk"]
    i = np.arange(cap)[None, :]
    inner = (i >= 1) & (i < Z[:, None] - 1)
    used = N[i < Z[:, None]].astype(np.int64)
    return {"stress": np.array(stress), "count": int(case["n"]), "hz": np.bincount(Z, minlength=cap + 2),
            "hn": np.bincount(used, minlength=cap + 2), "q": np.sort(ln[inner])}
