"""Timing cases of the framework: the work its users have it do, through the public entry points.

A case is a dict of plain values:
  kind     "g"        one equal-time G from device fields (hq_equaltime_g_noalloc)
           "sweep"    a round trip of update sweeps (0 -> beta -> 0) with the equal-time estimators
           "dynamic"  a time-displaced sweep and an update sweep back, with both sets of estimators
           "adjoint"  log|det(1 + B...B)| and its gradients for fixed fields
  L, beta, nt, pace, u, mu   lattice size, inverse temperature, slices, slices per stabilisation, |U|, mu
  chains   Markov chains in the context
  hop      "uniform" (separable exp(-dt K)), "dense" (the same K applied as a dense matrix) or
           "bonds" (a hopping of its own on every bond, set with set_hopping)
  mode     "launches" or "persistent": how a sweep is issued
  graph    whether the sweeps are replayed from captured CUDA graphs
  upload   whether a pass starts from fields in host memory (copy, stacks and G, sweeps, copy back)
  bin      round trips of a "dynamic" pass between two readings of the estimators
  uneven   chains of L = 6, 8, 10, 12, |U| = 2, 4, 6 and beta = 4, 8, 12 in one context
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

PKG = "hubbard-attractive-u_b200"
DEFAULTS = dict(kind="sweep", L=4, beta=4.0, nt=40, pace=10, u=4.0, mu=0.0, chains=1, hop="uniform",
                mode="launches", graph=False, upload=False, bin=1, uneven=False)
UP, DOWN, DYNAMIC, MEASURE = 0, 1, 2, 1


def _hq():
    name = "hubbard_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(PKG, "__init__.py"),
                                                      submodule_search_locations=[os.path.abspath(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def listed():
    return [
        # one Green's function of the smallest lattice, as a service calls it: launch latency
        dict(DEFAULTS, name="g_4x4", kind="g", beta=4.0, nt=40),
        # the plain single chain of the smallest configuration: launch latency of the sweep
        dict(DEFAULTS, name="chain_4x4", beta=4.0, nt=40),
        # the reference's example configuration with 64 chains (the command line's --chains 64):
        # equal-time and displaced observables, warm-up done
        dict(DEFAULTS, name="example_4x4_x64", kind="dynamic", beta=8.0, nt=160, chains=64, bin=4),
        # one chain with displaced G on all 160 slices
        dict(DEFAULTS, name="dynamic_8x8", kind="dynamic", L=8, beta=8.0, nt=160, mu=-0.5),
        # one chain of the benchmark's lattice: what a user with a single Markov chain gets
        dict(DEFAULTS, name="chain_12x12", L=12, beta=10.0, nt=100, graph=True),
        # an odd lattice and a ragged last interval, a third of the GPU's SMs busy
        dict(DEFAULTS, name="odd_9x9_x48", L=9, beta=4.7, nt=47, u=3.0, mu=0.2, chains=48),
        # hoppings of their own on every bond (disorder): the dense exp(-dt K), odd N
        dict(DEFAULTS, name="bonds_7x7_x32", L=7, beta=4.0, nt=40, chains=32, hop="bonds"),
        # gradients of the log-determinant of 64 fixed configurations
        dict(DEFAULTS, name="adjoint_10x10_x64", kind="adjoint", L=10, beta=6.0, nt=60, mu=-0.3, chains=64),
        # a lattice just too large for one SM's shared memory, few chains
        dict(DEFAULTS, name="mid_14x14_x16", L=14, beta=5.0, nt=50, chains=16),
        # the benchmark's workload end to end: fields from the host, stacks, a round trip, fields back
        dict(DEFAULTS, name="batch_12x12_x256", L=12, beta=10.0, nt=100, chains=256, graph=True, upload=True),
        # the batch of uneven chains, one persistent launch per sweep
        dict(DEFAULTS, name="uneven_x256", L=12, beta=12.0, nt=120, chains=256, uneven=True, mode="persistent", graph=True),
        # the large batched run: 64 chains whose G spans several SMs
        dict(DEFAULTS, name="large_16x16_x64", L=16, beta=16.0, nt=320, pace=8, mu=-0.2, chains=64, graph=True),
    ]


def draw(rng):
    kind = rng.choice(["g", "sweep", "sweep", "sweep", "dynamic", "adjoint"])
    pace = rng.choice([5, 8, 10, 10])
    c = dict(DEFAULTS, kind=kind, pace=pace, u=rng.choice([2.0, 3.0, 4.0, 6.0]), mu=rng.choice([0.0, -0.5, 0.25]))
    dt = 0.05 if rng.random() < 0.5 else 0.1
    c["L"] = rng.randint(3, {"g": 8, "sweep": 16, "dynamic": 12, "adjoint": 10}[kind])
    most = 16 * pace if kind == "g" else 160
    c["nt"] = int(round(math.exp(rng.uniform(math.log(pace + 1), math.log(most)))))
    c["beta"] = dt * c["nt"]
    if kind == "g":
        return c
    # chains over their logarithm, as many as keep the pass below the largest listed case
    weight = c["nt"] * max(c["L"], 4) ** 5 / (0.04 if c["L"] > 12 else 1.0)
    room = 2.0e9 if kind != "adjoint" else 4.0e8
    c["chains"] = int(round(math.exp(rng.uniform(0.0, math.log(max(1.0, min(256.0, room / weight)))))))
    c["hop"] = "uniform" if kind == "adjoint" or c["L"] > 12 else rng.choice(["uniform", "uniform", "dense", "bonds"])
    if kind == "dynamic":
        c["bin"] = rng.randint(1, 4)
    if kind == "sweep":
        c["mode"] = rng.choice(["launches", "persistent"]) if c["L"] <= 12 else "launches"
        c["graph"] = rng.random() < 0.5
        c["upload"] = rng.random() < 0.3
    return c


def _params(case, seed):
    n = int(case["chains"])
    expk = 0 if case["hop"] == "dense" else -1
    out = []
    for k in range(n):
        p = dict(nl=case["L"], nnt=1.0, u=case["u"], mu=case["mu"], beta=case["beta"], nt=case["nt"],
                 stabilization_pace=case["pace"], expk_mode=expk, seed=1000 + 1009 * seed + k,
                 dynamic=int(case["kind"] == "dynamic"))
        if case["uneven"]:
            p["nl"] = [6, 8, 10, 12][(k * 4) // n]
            p["u"] = [2.0, 4.0, 6.0][k % 3]
            p["beta"] = [4.0, 8.0, 12.0][(k // 3) % 3]
            p["nt"] = int(round(p["beta"] / 0.1))
        out.append(p)
    return out


def _neighbours(L):
    """Hopping matrix of the periodic lattice, site i = x + L y (bonds doubled at L = 2)."""
    h = np.zeros((L * L, L * L))
    for s in range(L * L):
        x, y = s % L, s // L
        for t in ((x + 1) % L + L * y, x + L * ((y + 1) % L)):
            h[s, t] += 1.0
            h[t, s] += 1.0
    return h


def _hopping(case, seed, k):
    h = _neighbours(case["L"])
    if case["hop"] != "bonds":
        return h
    r = np.random.RandomState((7919 * seed + k) % (1 << 31)).uniform(0.8, 1.2, h.shape)
    return h * np.triu(r) + (h * np.triu(r)).T - np.diag(np.diag(h * r))


def prepare(case, seed):
    hq = _hq()
    if case["kind"] == "g":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n2 = case["L"] ** 2
        f = (2 * torch.randint(0, 2, (case["nt"], n2), generator=g, device="cuda") - 1).to(torch.int8)
        return dict(case=case, lib=hq.lib(), check=hq.capi.check, fields=f,
                    g=torch.empty(n2, n2, dtype=torch.float64, device="cuda"))
    params = _params(case, seed)
    e = hq.Engine(params)
    if case["hop"] == "bonds":
        for k in range(e.n):
            e.set_hopping(k, _hopping(case, seed, k))
    if case["mode"] == "persistent":
        e.set_sweep_mode(hq.SWEEP_PERSISTENT)
    e.fields_random()
    host = torch.empty(sum(p["nt"] * p["nl"] ** 2 for p in params), dtype=torch.int8, pin_memory=True)
    e.download_fields_i8(host.data_ptr())
    e.sync()
    if case["kind"] != "adjoint":
        e.init()
    if case["graph"]:
        e.capture_graph(UP, MEASURE)
        e.capture_graph(DOWN, MEASURE)
    return dict(case=case, e=e, host=host)


def _looked_at(n):
    """The chains whose updated G a pass reads back: every one where there are few; a large
    batch's stay on the device, where the next sweep needs them."""
    return range(n) if n <= 16 else (0, n - 1)


def run(state):
    case = state["case"]
    if case["kind"] == "g":
        state["check"](state["lib"].hq_equaltime_g_noalloc(
            case["L"], 1.0, case["u"], case["mu"], case["beta"], case["nt"], case["pace"], state["fields"].data_ptr(),
            state["g"].data_ptr(), torch.cuda.current_stream().cuda_stream))
        return {"g": state["g"]}
    e, host = state["e"], state["host"]
    if case["kind"] == "adjoint":
        e.init()  # the pass leaves the stacks at tau = beta
        logdet, grads = e.logdet_adjoint()
        return {"logdet": logdet, "dmu": np.array([x[0] for x in grads]), "dalpha": np.array([x[1] for x in grads]),
                "dK": np.stack([x[2] for x in grads])}
    if case["kind"] == "dynamic":
        e.reset_estimators()
        for _ in range(case["bin"]):
            e.sweep(DYNAMIC)
            e.sweep(DOWN, MEASURE)
        e.sync()
        est = e.estimators_all()
        dyn = [e.dynamic_estimators(k) for k in range(e.n)]
        return {"estimators": est, "g": [e.g(k) for k in _looked_at(e.n)], "spin": np.stack([d[0] for d in dyn]), "ldos": np.stack([d[1] for d in dyn]),
                "gd": np.stack([d[2] for d in dyn])}
    if case["upload"]:
        e.upload_fields_i8(host.data_ptr())
        e.init()
    e.sweep(UP, MEASURE)
    e.sweep(DOWN, MEASURE)
    e.download_fields_i8(host.data_ptr())
    est = e.estimators_all()  # waits for the sweeps and the copy
    return {"fields": host, "estimators": est, "g": [e.g(k) for k in _looked_at(e.n)]}


def work(case):
    """What a pass cannot do without: the separable (or dense) exp(-dt K) products of the wraps
    and B chains, two multiply-adds per element and accepted flip (about 0.64 of the proposals),
    and per stabilisation the factorisation, its V^T, the builder's products and its inverse;
    fields, G and stack entries read and written once."""
    flops = nbytes = 0.0
    for p in _params(dict(case, chains=max(1, case["chains"])), 0):
        L, N, nt = p["nl"], p["nl"] ** 2, p["nt"]
        ns = -(-nt // p["stabilization_pace"])
        expk = 4.0 * N * L ** 3 if case["hop"] == "uniform" and L <= 16 else 2.0 * N ** 3  # one application
        push = (8.0 / 3.0 + 2.0) * N ** 3
        build = 10.0 * N ** 3
        entry = 8.0 * (2 * N * N + N)
        init = nt * expk + ns * push + build
        if case["kind"] == "g":
            flops += init
            nbytes += nt * N + 8.0 * N * N
            continue
        updates = nt * (2 * expk + 0.64 * N * 2.0 * N * N)
        one_way = nt * expk + updates + ns * (push + build)
        if case["kind"] == "sweep":
            flops += 2 * one_way + (init if case["upload"] else 0.0)
            nbytes += 2 * (2.0 * nt * N + 16.0 * N * N + 2 * ns * entry)
        elif case["kind"] == "dynamic":
            flops += case["bin"] * (one_way + 5 * nt * expk + ns * (push + build + 6.0 * N ** 3))
            nbytes += case["bin"] * 2 * (2.0 * nt * N + 16.0 * N * N + 2 * ns * entry) + 8.0 * (2 + N) * nt
        else:
            flops += init + 2 * nt * expk + nt * expk + nt * 2.0 * N * N + ns * (push + build) + 14.0 * N ** 3
            nbytes += nt * N + 8.0 * N * N + 2 * ns * entry
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------
#  The same outputs in plain torch, 64 bits: the chains in lockstep, G rebuilt from the block
#  matrix of the imaginary-time path every `pace` slices.
# ---------------------------------------------------------------------------------------------
M31 = 2147483647


def _uniforms(seeds, skip, count):
    """Draws skip .. skip + count - 1 of each chain's stream (minstd_rand0, two values a draw)."""
    x = np.array([s % M31 or 1 for s in seeds], dtype=np.uint64)
    x = x * np.uint64(pow(16807, 2 * skip, M31)) % np.uint64(M31)
    out = np.empty((count, len(seeds)))
    R = 2147483646.0
    for k in range(count):
        x1 = x * np.uint64(16807) % np.uint64(M31)
        x = x1 * np.uint64(16807) % np.uint64(M31)
        out[k] = ((x1 - np.uint64(1)).astype(np.float64) + (x - np.uint64(1)).astype(np.float64) * R) / (R * R)
    return torch.from_numpy(np.minimum(out, np.nextafter(1.0, 0.0)))


class _Exact:
    def __init__(self, case, hop, fields):
        """hop: [n][N][N], fields: [n][nt][N] of +-1 (doubles)."""
        self.c, self.f = case, fields
        self.n, self.nt, self.N = fields.shape
        dt = case["beta"] / case["nt"]
        self.alpha = math.acosh(math.exp(0.5 * dt * case["u"]))
        K = -hop - case["mu"] * torch.eye(self.N, dtype=torch.float64, device=hop.device)
        self.dt, self.K = dt, K
        w, Q = torch.linalg.eigh(K)
        self.w, self.Q = w, Q
        self.E = (Q * torch.exp(-dt * w)[:, None, :]) @ Q.mT
        self.Ei = (Q * torch.exp(dt * w)[:, None, :]) @ Q.mT
        self.eye = torch.eye(self.N, dtype=torch.float64, device=hop.device)

    def B(self, l, M):
        return torch.exp(self.alpha * self.f[:, l % self.nt])[:, :, None] * (self.E @ M)

    def up(self, l, G):
        v = torch.exp(self.alpha * self.f[:, l % self.nt])
        return v[:, :, None] * (self.E @ G @ self.Ei) / v[:, None, :]

    def down(self, l, G):
        v = torch.exp(self.alpha * self.f[:, l % self.nt])
        return self.Ei @ (G / v[:, :, None] * v[:, None, :]) @ self.E

    def matrix(self, t):
        """The block matrix whose inverse holds G between the slices t, t + pace, ...: blocks of
        at most `pace` slices each, starting after slice t."""
        starts = list(range(0, self.nt, self.c["pace"])) + [self.nt]
        k = len(starts) - 1
        N = self.N
        A = torch.eye(k * N, dtype=torch.float64, device=self.E.device).repeat(self.n, 1, 1)
        for b in range(k):
            P = self.eye.repeat(self.n, 1, 1)
            for l in range(starts[b], starts[b + 1]):
                P = self.B(t + 1 + l, P)
            r = (b + 1) % k
            A[:, r * N:(r + 1) * N, b * N:(b + 1) * N] += P if r == 0 else -P
        return A, starts

    def G(self, t):
        A, _ = self.matrix(t)
        rhs = torch.zeros(self.n, A.shape[1], self.N, dtype=torch.float64, device=A.device)
        rhs[:, :self.N] = self.eye
        return torch.linalg.solve(A, rhs)[:, :self.N]

    def flips(self, l, G, u):
        """Metropolis visits of slice l in site order; u: [N][n] uniforms. Returns G, flips."""
        s = self.f[:, l]
        count = torch.zeros(self.n, dtype=torch.float64, device=G.device)
        d = torch.exp(-2 * self.alpha * s) - 1.0
        for i in range(self.N):
            a = 1.0 + (1.0 - G[:, i, i]) * d[:, i]
            acc = u[i] < (a * a / (1.0 + d[:, i])).abs()
            row = -G[:, i, :]
            row[:, i] += 1.0
            col = G[:, :, i] * torch.where(acc, d[:, i] / a, torch.zeros_like(a))[:, None]
            G = torch.baddbmm(G, col[:, :, None], row[:, None, :], alpha=-1.0)
            s[:, i] = torch.where(acc, -s[:, i], s[:, i])
            count += acc
        return G, count

    def sweep(self, direction, G, u, est):
        nt, N, pace = self.nt, self.N, self.c["pace"]
        for k in range(nt):
            t = k + 1 if direction == UP else nt - k
            if direction == UP:
                G, c = self.flips(t % nt, self.up(t, G), u[k * N:(k + 1) * N])
                if t % pace == 0 or t == nt:
                    G = self.G(t)
            else:
                G, c = self.flips(t % nt, G, u[k * N:(k + 1) * N])
                G = self.G(t - 1) if (t - 1) % pace == 0 else self.down(t, G)
            tr = G.diagonal(dim1=1, dim2=2).sum(1)
            est[:, 0] += 2.0 - 2.0 * tr / N
            est[:, 1] += (1.0 - G.diagonal(dim1=1, dim2=2)).square().sum(1) / N
            est[:, 2] += (2.0 * G.square().sum((1, 2)) - 2.0 * tr + N) / N
            est[:, 3] += 1.0
            est[:, 4] += N
            est[:, 5] += c
        return G

    def displaced(self):
        """spin[nt], ldos[nt], gd[N][nt] of every chain from G(tau, 0) and G(0, tau)."""
        nt, N, L = self.nt, self.N, self.c["L"]
        A, starts = self.matrix(0)
        inv = torch.linalg.inv(A)
        spin = torch.zeros(self.n, nt, dtype=torch.float64, device=A.device)
        ldos, gd = torch.zeros_like(spin), torch.zeros(self.n, N, nt, dtype=torch.float64, device=A.device)
        d, i = np.arange(N)[:, None], np.arange(N)[None, :]
        j = torch.from_numpy((i % L + d % L) % L + L * ((i // L + d // L) % L)).to(A.device)
        i = torch.arange(N, device=A.device).expand(N, N)
        for b in range(len(starts) - 1):
            t0 = inv[:, b * N:(b + 1) * N, :N]
            zt = inv[:, :N, b * N:(b + 1) * N] - (self.eye if b == 0 else 0.0)
            for l in range(starts[b], starts[b + 1]):
                if l > starts[b]:
                    v = torch.exp(self.alpha * self.f[:, l])
                    t0 = self.B(l, t0)
                    zt = (zt @ self.Ei) / v[:, None, :]
                x, y = t0.diagonal(dim1=1, dim2=2), zt.diagonal(dim1=1, dim2=2)
                spin[:, l] = -(x * y).sum(1) / N
                ldos[:, l] = x.sum(1) / N
                gd[:, :, l] = t0[:, j, i].sum(2)
        return spin, ldos, gd

    def gradients(self):
        """log|det|, d/dmu, d/dalpha and d/dK of every chain."""
        nt, N = self.nt, self.N
        n, dev = self.n, self.E.device
        dmu, dal = torch.zeros(n, dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev)
        D = torch.zeros(n, N, N, dtype=torch.float64, device=dev)
        G = self.G(0)
        logdet = torch.linalg.slogdet(self.matrix(0)[0])[1]
        for t in range(1, nt + 1):
            G = self.G(t) if t % self.c["pace"] == 0 or t == nt else self.up(t, G)
            one = self.eye - G
            s = self.f[:, t % nt]
            dmu += self.dt * one.diagonal(dim1=1, dim2=2).sum(1)
            dal += (s * one.diagonal(dim1=1, dim2=2)).sum(1)
            v = torch.exp(self.alpha * s)
            D += one / v[:, :, None] * v[:, None, :]
        Mt = self.Q.mT @ (self.Ei @ D) @ self.Q
        f = torch.exp(-self.dt * self.w)
        dw = self.w[:, :, None] - self.w[:, None, :]
        same = dw.abs() <= 1e-10
        div = torch.where(same, -self.dt * 0.5 * (f[:, :, None] + f[:, None, :]),
                          (f[:, :, None] - f[:, None, :]) / torch.where(same, torch.ones_like(dw), dw))
        return logdet, dmu, dal, self.Q @ (div * Mt.mT) @ self.Q.mT


def exact(case, seed):
    if case["uneven"]:
        return None
    n, nt, N, pace = max(1, case["chains"]), case["nt"], case["L"] ** 2, case["pace"]
    order = -(-nt // pace) * N
    builds = {"g": 1, "adjoint": -(-nt // pace), "dynamic": case["bin"] * (3 - (-nt // pace)), "sweep": 2 * -(-nt // pace)}[case["kind"]]
    sites = {"g": 0, "adjoint": 0, "dynamic": case["bin"], "sweep": 2}[case["kind"]] * nt * N
    # seconds on one GPU, roughly: the block solves (one matrix at a time) and the site visits
    if builds * n * (3e-4 + 2.5e-12 * order ** 3) + 1.2e-4 * sites > 15.0 or 24.0 * n * order ** 2 > 4e10:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cpu = lambda x: x.cpu().numpy()  # noqa: E731
    if case["kind"] == "g":
        g = torch.Generator(device=dev).manual_seed(seed)
        f = (2 * torch.randint(0, 2, (nt, N), generator=g, device=dev) - 1).double()
        x = _Exact(case, torch.from_numpy(_neighbours(case["L"])).to(dev)[None], f[None])
        return {"g": x.G(0)[0].mT.contiguous()}  # column-major
    seeds = [p["seed"] for p in _params(case, seed)]
    f = torch.where(_uniforms(seeds, 0, nt * N) < 0.5, 1.0, -1.0).double().T.reshape(n, nt, N).contiguous().to(dev)
    hop = torch.from_numpy(np.stack([_hopping(case, seed, k) for k in range(n)])).to(dev)
    x = _Exact(case, hop, f)
    if case["kind"] == "adjoint":
        logdet, dmu, dal, dK = x.gradients()
        return {"logdet": cpu(logdet), "dmu": cpu(dmu), "dalpha": cpu(dal), "dK": cpu(dK)}
    est = torch.zeros(n, 6, dtype=torch.float64, device=dev)
    if case["kind"] == "dynamic":
        u = _uniforms(seeds, nt * N, case["bin"] * nt * N).to(dev)
        spin = ldos = gd = 0.0
        for k in range(case["bin"]):
            spin, ldos, gd = (a + b for a, b in zip((spin, ldos, gd), x.displaced()))
            G = x.sweep(DOWN, x.G(0), u[k * nt * N:(k + 1) * nt * N], est)
        return {"estimators": cpu(est), "g": [cpu(G[k]) for k in _looked_at(n)], "spin": cpu(spin), "ldos": cpu(ldos), "gd": cpu(gd)}
    u = _uniforms(seeds, nt * N, 2 * nt * N).to(dev)
    G = x.sweep(UP, x.G(0), u[:nt * N], est)
    G = x.sweep(DOWN, G, u[nt * N:], est)
    return {"fields": None, "estimators": cpu(est), "g": [cpu(G[k]) for k in _looked_at(n)]}
