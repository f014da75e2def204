"""What the framework is timed on: bins of Markov chains, alone and in batches,
the time-displaced and global passes, the adjoint and the module procedures,
each through the public host API (``z2_gauge_zfy_b200``).

A case lists the lattices ("LXxLY,...") and the numbers of time slices
("L1,L2,...") of its chains: chain i takes lattice i mod (number of lattices)
and slices entry (i div number of lattices) mod (number of entries).  ``h`` is
drawn per chain from [h_lo, h_hi]; seeds of chains and couplings come from the
case's seed.  ``call`` names the pass:

  bin      Z2Batch.sweep (one bin of every chain) and the bin's observables
  tau      the same with the time-displaced pass, and the correlators
  global   Wolff-in-tau moves, then a bin (the reference's recorded run)
  adjoint  Z2Batch.logdet_grad
  modules  a stabilization interval driven procedure by procedure on host
           matrices: OperatorKin%mmult_R per slice, stab_UR, stab_green

Every size keeps dtau * slices = beta, and slices are multiples of nwrap.
"""
import math
import random

import numpy as np

from z2_gauge_zfy_b200 import Chain, Z2Batch

# Chains of a handle whose matrices are read back after a pass: all of a small
# handle; one of each (lattice, slices) class of a large batch.
READ_ALL = 8


def _case(name, call, lattices, slices, chains, **more):
    c = {"name": name, "call": call, "lattices": lattices, "slices": slices, "chains": chains,
         "dtau": 0.1, "nwrap": 10, "J": 0.5, "h_lo": 0.5, "h_hi": 0.5, "mu": 0.0, "t": 1.0,
         "start": 1, "delay": 0, "exact_pivots": False, "nglobal": 0}
    c.update(more)
    return c


def listed():
    return [
        # the CPU-runnable plain configuration: a test run, a first look at a
        # parameter set; the smallest launch, all latency
        _case("bin_4x4", "bin", "4x4", "40", 1),
        # plain DQMC on the GPU: one chain, equal-time observables each bin
        _case("bin_8x8", "bin", "8x8", "100", 1),
        # one chain of the largest lattice that fits a multiprocessor's shared
        # memory at low temperature: a user following a single parameter point
        _case("bin_12x12", "bin", "12x12", "160", 1),
        # the headline workload: a scan over sizes, temperatures and fields in
        # one launch
        _case("bins_256_uneven", "bin", "6x6,8x8,10x10,12x12", "80,120,160", 256,
              h_lo=0.2, h_hi=1.0),
        # many replicas of small lattices: error bars, tempering-style scans
        _case("bins_512_small", "bin", "4x4,6x6", "40,80", 512, h_lo=0.2, h_hi=1.0),
        # rectangular lattices away from half filling (finite-size checks)
        _case("bins_24_rect_mu", "bin", "4x6,6x10,8x12,10x14", "60", 24, mu=0.3, h_lo=0.4,
              h_hi=0.8),
        # the reference's column pivoting, for runs compared with the Fortran
        # program factor by factor
        _case("bins_16_exact_pivots", "bin", "8x8", "80", 16, exact_pivots=True),
        # the large production lattice with the time-displaced pass and the
        # momentum-space correlators (shorter than a production beta)
        _case("tau_8_16x16", "tau", "16x16", "64", 8, dtau=0.05, nwrap=8, h_lo=0.6, h_hi=0.6,
              delay=32),
        # one chain with the time-displaced pass
        _case("tau_10x10", "tau", "10x10", "80", 1),
        # the reference's recorded run (test_run): global moves before each bin
        _case("global_16_4x4", "global", "4x4", "40", 16, dtau=0.05, nwrap=5, J=1.0, h_lo=0.52,
              h_hi=0.52, mu=0.3, t=0.5, start=5, nglobal=4),
        # gradient of log det with respect to every hopping and mu
        _case("adjoint_12x12", "adjoint", "12x12", "120", 1, mu=0.1),
        # a host program that keeps its own loop and calls the module
        # procedures on its own matrices
        _case("modules_10x10", "modules", "10x10", "40", 2),
    ]


def _even(rng, lo, hi):
    """An even number in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1.99)))
    return max(lo, min(hi, int(v) // 2 * 2))


def draw(rng):
    call = rng.choice(["bin", "bin", "bin", "bin", "tau", "tau", "global", "adjoint", "modules"])
    nwrap = rng.choice([5, 8, 10])
    dtau = rng.choice([0.05, 0.1])
    more = {"dtau": dtau, "nwrap": nwrap, "mu": rng.choice([0.0, 0.0, round(rng.uniform(-0.5, 0.5), 3)]),
            "J": round(rng.uniform(0.3, 1.0), 3), "h_lo": 0.2, "h_hi": 1.0,
            "t": round(rng.uniform(0.5, 1.0), 3), "start": rng.choice([1, 1, 2, 5])}
    wraps = rng.randint(4, 16)
    if call == "bin":
        chains = max(1, int(math.exp(rng.uniform(0.0, math.log(512.0)))))
        nlat = rng.randint(1, 4) if chains > 1 else 1
        lat = ["%dx%d" % ((n, n) if rng.random() < 0.6 else (n, _even(rng, 4, 12)))
               for n in (_even(rng, 4, 12) for _ in range(nlat))]
        if chains == 1 and rng.random() < 0.2:
            lat, wraps = [rng.choice(["14x14", "12x16", "16x16"])], 6
        # no more work than the headline batch
        big = max(int(a) * int(b) for a, b in (s.split("x") for s in lat))
        chains = max(1, min(chains, int(2.7e8 / (big * big * nwrap * wraps))))
        more["exact_pivots"] = rng.random() < 0.15
        return _strip(_case("", call, ",".join(lat), str(nwrap * wraps), chains, **more))
    if call == "tau":
        n = _even(rng, 4, 12)
        return _strip(_case("", call, "%dx%d" % (n, n), str(nwrap * rng.randint(3, 8)),
                            rng.randint(1, 8), **more))
    if call == "global":
        n = _even(rng, 4, 8)
        return _strip(_case("", call, "%dx%d" % (n, n), str(nwrap * rng.randint(4, 8)),
                            rng.randint(1, 32), nglobal=rng.randint(1, 4), **more))
    more["mu"] = round(rng.uniform(-0.3, 0.3), 3)
    n, m = _even(rng, 4, 12), _even(rng, 4, 12)
    if call == "adjoint":
        return _strip(_case("", call, "%dx%d" % (n, m), str(nwrap * wraps), 1, **more))
    return _strip(_case("", call, "%dx%d" % (n, m), str(nwrap * rng.randint(2, 6)), 2, **more))


def _strip(c):
    del c["name"]
    return c


# ---------------------------------------------------------------------------
def _chain_params(case, seed):
    rng = random.Random(1000003 * int(seed) + 17)
    lats = [tuple(int(v) for v in s.split("x")) for s in case["lattices"].split(",")]
    sl = [int(v) for v in case["slices"].split(",")]
    out = []
    for i in range(case["chains"]):
        lx, ly = lats[i % len(lats)]
        lt = sl[(i // len(lats)) % len(sl)]
        h = rng.uniform(case["h_lo"], case["h_hi"])
        s = rng.randrange(1, 2 ** 30) | 1
        rt = None
        if case["call"] == "adjoint":
            rt = case["t"] * (1.0 + 0.05 * np.random.default_rng(s).standard_normal(2 * lx * ly))
        out.append(dict(RT=case["t"], J=case["J"], h=h, mu=case["mu"], Nlx=lx, Nly=ly, Ltrot=lt,
                        beta=case["dtau"] * lt, Nwrap=case["nwrap"], absolute=case["start"],
                        seed=s, rt_bond=rt))
    return out


def _read(case):
    """Chains whose links and Green's function are read back after a pass."""
    n = case["chains"]
    if n <= READ_ALL:
        return list(range(n))
    classes = len(case["lattices"].split(",")) * len(case["slices"].split(","))
    return list(range(min(n, classes)))


def prepare(case, seed):
    """The handle a program keeps across its run: chains created from their
    seeds, the first Green's function computed (``Local_sweep_pre``)."""
    par = _chain_params(case, seed)
    b = Z2Batch([Chain(**p) for p in par], delay_k=case["delay"], tau=case["call"] == "tau",
                stab_exact=case["exact_pivots"])
    if case["call"] == "adjoint":
        return {"case": case, "batch": b}
    b.pre()
    s = {"case": case, "batch": b}
    if case["call"] == "modules":
        s.update(_module_inputs(case, par))
    return s


def _module_inputs(case, par):
    """UDV factors as the path meets them, formed by numpy: the right product
    from chain 0's links, the left one from the transpose of chain 1's."""
    (U, D, V), (u, d, v) = (_Model(p, case["dtau"]).udv(0) for p in par[:2])
    return {"UR": U, "DR": D, "VR": V, "UL": u.T.copy(), "DL": d, "VL": v.T.copy()}


def _outputs(case, b):
    out = {"obs": b.obs_equal_all()}
    for i in _read(case):
        sigma, iseed = b.get_config(i)
        out["chain%d" % i] = {"sigma": sigma.astype(np.int8), "seed": iseed, "G": b.green(i)}
    return out


def run(state):
    case, b = state["case"], state["batch"]
    call = case["call"]
    if call == "bin":
        b.sweep(1)
        return _outputs(case, b)
    if call == "tau":
        b.sweep(1, toggle=True)
        out = _outputs(case, b)
        for i in range(case["chains"]):
            k = b.obs_tau_k(i)
            out["tau%d" % i] = np.stack([k[q] for q in sorted(k)])
        return out
    if call == "global":
        b.sweep_global(case["nglobal"])
        b.sweep(1)
        return _outputs(case, b)
    if call == "adjoint":
        ld, grad, dmu = b.logdet_grad(0)
        return {"logdet": ld, "grad": grad, "dmu": dmu}
    U = state["UR"]
    for nt in range(1, case["nwrap"] + 1):
        U = b.opk_mmult_R(0, U, nt, 1)
    U, D, V = b.stab_UR(0, U, state["DR"], state["VR"])
    G = b.stab_green(0, U, D, V, state["UL"], state["DL"], state["VL"], case["nwrap"])
    return {"U": U, "D": D, "V": V, "G": G}


def work(case):
    """Per site-update (one site of one slice of a half-sweep): 72 N flops of
    checkerboard wraps, 8 a N^2 of rank-2 updates (acceptance a = 0.1), 14
    N^2 / nwrap of stabilization and 20 N of observables; the time-displaced
    pass and a global move add a half-sweep's wraps and stabilization.  Bytes:
    the links, Green's function and the UDV factors at every interval, read
    and written once."""
    flops = byt = 0.0
    for p in _chain_params(case, 0):
        n, lt, w = p["Nlx"] * p["Nly"], p["Ltrot"], p["Nwrap"]
        half = n * lt
        wraps = 72.0 * n + 14.0 * n * n / w
        if case["call"] == "modules":
            flops += 36.0 * n * n * w + 14.0 * n ** 3
            byt += 8.0 * n * n * 10
            break
        if case["call"] == "adjoint":
            flops += 3 * half * wraps
        else:
            flops += 2 * half * (wraps + 0.8 * n * n + 20.0 * n)
            if case["call"] == "tau":
                flops += half * (2 * wraps + 14.0 * n * n / w + 40.0 * n)
            flops += case["nglobal"] * half * wraps
        byt += 2.0 * (2 * n * lt + 8.0 * n * n * (1 + 2 * (lt // w)))
        if case["call"] == "tau":
            byt += 16.0 * 7 * lt * n
    return {"bytes": byt, "flops": flops}


# ---------------------------------------------------------------------------
# The same passes in plain numpy (float64): links from their seeds, dense
# Green's functions, one proposal after the other.
# ---------------------------------------------------------------------------
class _Model:
    def __init__(self, p, dtau):
        self.p, self.dtau = p, dtau
        lx, ly = p["Nlx"], p["Nly"]
        self.n = n = lx * ly
        self.nb, self.lt = 2 * n, p["Ltrot"]
        site = lambda x, y: (y % ly) * lx + x % lx  # noqa: E731
        self.xy = [(s % lx, s // lx) for s in range(n)]
        self.bonds = np.zeros((2 * n, 2), dtype=int)
        self.plaq = np.zeros((2 * n, 6), dtype=int)     # two plaquettes of a bond, the other bonds
        self.face = np.zeros((n, 4), dtype=int)
        X = lambda x, y: 2 * site(x, y)  # noqa: E731
        Y = lambda x, y: 2 * site(x, y) + 1  # noqa: E731
        groups = [[], [], [], []]
        for s, (x, y) in enumerate(self.xy):
            self.bonds[2 * s] = s, site(x + 1, y)
            self.bonds[2 * s + 1] = s, site(x, y + 1)
            up = (Y(x, y), X(x, y + 1), Y(x + 1, y))
            self.plaq[2 * s] = up + (Y(x, y - 1), X(x, y - 1), Y(x + 1, y - 1))
            self.plaq[2 * s + 1] = (X(x, y), Y(x + 1, y), X(x, y + 1),
                                    X(x - 1, y), Y(x - 1, y), X(x - 1, y + 1))
            self.face[s] = X(x, y), Y(x + 1, y), X(x, y + 1), Y(x, y)
            groups[0 if x % 2 else 1].append(2 * s)
            groups[2 if y % 2 else 3].append(2 * s + 1)
        self.groups = [np.array(g) for g in groups]
        rt = p["rt_bond"] if p["rt_bond"] is not None else np.full(2 * n, p["RT"])
        self.rt = np.asarray(rt, dtype=float)
        self.ch, self.sh = np.cosh(0.5 * dtau * self.rt), np.sinh(0.5 * dtau * self.rt)
        self.mu = math.exp(dtau * p["mu"])
        self.order = [0, 1, 2, 3, 3, 2, 1, 0]
        self.state = p["seed"]
        self.links()

    def ranf(self):
        self.state = (self.state * 48828125) % 2 ** 31
        return self.state / 2.0 ** 31

    def links(self):
        n, nb, lt, kind = self.n, self.nb, self.lt, self.p["absolute"]
        s = np.ones((lt, nb))
        if kind == 1:
            s = np.array([[1.0 if self.ranf() >= 0.5 else -1.0 for _ in range(nb)] for _ in range(lt)])
        elif kind == 2:
            for t in range(lt):
                for b in range(nb):
                    a, c = self.ranf(), self.ranf()
                    v = math.sqrt(-2.0 * math.log(a)) * math.cos(2.0 * math.pi * c)
                    s[t, b] = 1.0 if v >= 0.0 else -1.0
        elif kind == 5:
            s[:] = np.array([1.0 if self.ranf() >= 0.5 else -1.0 for _ in range(nb)])
        for _ in range(n):
            self.ranf()
        self.sigma = s

    def rot(self, M, t, g, sign, rows):
        b = self.groups[g]
        i, j = self.bonds[b, 0], self.bonds[b, 1]
        C, S = self.ch[b], sign * self.sigma[t, b] * self.sh[b]
        if rows:
            a, c = M[i], M[j]
            M[i], M[j] = C[:, None] * a + S[:, None] * c, S[:, None] * a + C[:, None] * c
        else:
            a, c = M[:, i], M[:, j]
            M[:, i], M[:, j] = a * C + c * S, a * S + c * C

    def kin(self, M, t, sign, rows):
        for g in self.order:
            self.rot(M, t, g, sign, rows)

    def udv(self, nt):
        """B_nt ... B_1 B_Ltrot ... B_nt+1 = U D V (V well conditioned)."""
        n, w, lt = self.n, self.p["Nwrap"], self.lt
        U, D, V = np.eye(n), np.ones(n), np.eye(n)
        ts = [(nt + k) % lt for k in range(lt)]
        for c in range(0, lt, w):
            for t in ts[c:c + w]:
                self.kin(U, t, 1, True)
                U *= self.mu
            A = U * D
            q = np.argsort(-np.linalg.norm(A, axis=0), kind="stable")
            U, R = np.linalg.qr(A[:, q])
            D = np.abs(np.diag(R))
            V = (R / D[:, None]) @ V[q]
        return U, D, V

    def green(self, nt):
        U, D, V = self.udv(nt)
        Db, Ds = np.maximum(D, 1.0), np.minimum(D, 1.0)
        return np.linalg.solve(U.T / Db[:, None] + Ds[:, None] * V, U.T / Db[:, None])

    def propose(self, G, t, order):
        p, sig, lt = self.p, self.sigma, self.lt
        before, after, now = sig[(t - 1) % lt], sig[(t + 1) % lt], sig[t]
        gamma = -0.5 * math.log(math.tanh(self.dtau * p["h"]))
        for b in order:
            i, j = self.bonds[b]
            s = now[b]
            a2 = self.dtau * self.rt[b]
            co, si, so = math.cosh(a2), math.sinh(a2), math.sinh(-a2)
            d11 = co * co - si * so - 1.0
            d12 = -s * (si * co - co * so)
            l11, l12, l21, l22 = 1.0 - G[i, i], -G[i, j], -G[j, i], 1.0 - G[j, j]
            p11, p12 = 1.0 + d11 * l11 + d12 * l21, d11 * l12 + d12 * l22
            p21, p22 = d12 * l11 + d11 * l21, 1.0 + d12 * l12 + d11 * l22
            det = p11 * p22 - p12 * p21
            q = self.plaq[b]
            w = s * (now[q[0]] * now[q[1]] * now[q[2]] + now[q[3]] * now[q[4]] * now[q[5]])
            v = s * (before[b] + after[b])
            ratio = det * det * math.exp(self.dtau * p["J"] * -2.0 * w) * math.exp(gamma * -2.0 * v)
            if abs(ratio) > self.ranf():
                u = G[:, [i, j]] @ (np.array([[p22, -p12], [-p21, p11]]) / det)
                y = -G[[i, j]]
                y[0, i] += 1.0
                y[1, j] += 1.0
                G -= u @ (np.array([[d11, d12], [d12, d11]]) @ y)
                now[b] = -s

    def measure(self, G, t, acc):
        n, p = self.n, self.p
        flux = float(np.prod(self.sigma[t][self.face], axis=1).sum()) / n
        ni = 1.0 - np.diag(G)
        d = np.eye(n)
        a = np.outer(ni, ni)
        dc = 4.0 * a - 2.0 * (d - G.T) * G
        st = np.array([1.0 if (x + y) % 2 == 0 else -1.0 for x, y in self.xy])
        qx = math.pi - 2.0 * math.pi / p["Nlx"]
        x, y = np.array(self.xy).T
        ph = np.cos(qx * (x[:, None] - x[None]) + math.pi * (y[:, None] - y[None]))
        acc += [flux, flux * flux, ((d - G) ** 2).sum(), (np.outer(st, st) * dc).sum(),
                (ph * dc).sum(), 2.0 * ni.sum() / n, 1.0]

    def bin(self):
        n, w, lt = self.n, self.p["Nwrap"], self.lt
        acc = np.zeros(7)
        G = self.green(0)
        for nt in range(lt, 0, -1):
            if nt % w == 0 and nt != lt:
                G = self.green(nt)
            self.measure(G, nt - 1, acc)
            self.propose(G, nt - 1, range(self.nb - 1, -1, -1))
            self.kin(G, nt - 1, 1, False)
            self.kin(G, nt - 1, -1, True)
        G = self.green(0)
        for nt in range(1, lt + 1):
            self.kin(G, nt - 1, 1, True)
            self.kin(G, nt - 1, -1, False)
            self.propose(G, nt - 1, range(self.nb))
            if nt % w == 0:
                G = self.green(nt % lt)
            self.measure(G, nt - 1, acc)
        m = acc[:6] / acc[6]
        o = [m[0], self.p["beta"] * n * max(0.0, m[1] - m[0] ** 2), m[2] / n, m[3] / n, m[4] / n, 0.0, m[5]]
        o[5] = 1.0 - o[4] / o[3] if o[3] > 1.0e-12 else 0.0
        return np.array(o), G

    def logdet_grad(self):
        U, D, V = self.udv(0)
        Db, Ds = np.maximum(D, 1.0), np.minimum(D, 1.0)
        ld = float(np.log(Db).sum() + np.linalg.slogdet(U.T / Db[:, None] + Ds[:, None] * V)[1])
        grad = np.zeros(self.nb)
        dmu = 0.0
        for nt in range(self.lt):
            if nt % self.p["Nwrap"] == 0:
                G = self.green(nt)
                if nt == 0:
                    dmu = self.p["beta"] * float((1.0 - np.diag(G)).sum())
            for g in self.order:
                b = self.groups[g]
                i, j = self.bonds[b, 0], self.bonds[b, 1]
                grad[b] -= 0.5 * self.dtau * self.sigma[nt, b] * (G[i, j] + G[j, i])
                self.rot(G, nt, g, 1, True)
                self.rot(G, nt, g, -1, False)
        return ld, grad, dmu


def _pivoted_qr(A):
    """Householder QR with column pivoting: Q, R, pivots."""
    A = A.copy()
    n = A.shape[0]
    Q, piv = np.eye(n), np.arange(n)
    for k in range(n):
        m = k + int(np.argmax(np.linalg.norm(A[k:, k:], axis=0)))
        A[:, [k, m]], piv[[k, m]] = A[:, [m, k]], piv[[m, k]]
        v = A[k:, k].copy()
        if k == n - 1 or not np.any(v[1:]):
            continue
        v[0] += math.copysign(float(np.linalg.norm(v)), v[0])
        v /= np.linalg.norm(v)
        A[k:] -= 2.0 * np.outer(v, v @ A[k:])
        Q[:, k:] -= 2.0 * np.outer(Q[:, k:] @ v, v)
    return Q, np.triu(A), piv


def exact(case, seed):
    call = case["call"]
    par = _chain_params(case, seed)
    if call == "modules":
        s = _module_inputs(case, par)
        m = _Model(par[0], case["dtau"])
        U = s["UR"].copy()
        for t in range(case["nwrap"]):
            m.kin(U, t, 1, True)
        Q, R, piv = _pivoted_qr(U * s["DR"])
        D = np.abs(np.diag(R))
        V = (R / D[:, None]) @ s["VR"][piv]
        Rb, Rs = np.maximum(D, 1.0), np.minimum(D, 1.0)
        Lb, Ls = np.maximum(s["DL"], 1.0), np.minimum(s["DL"], 1.0)
        M = (Q.T @ s["UL"].T) / Rb[:, None] / Lb + Rs[:, None] * (V @ s["VL"]) * Ls
        G = (s["UL"].T / Lb) @ np.linalg.solve(M, Q.T / Rb[:, None])
        return {"U": Q, "D": D, "V": V, "G": G}
    if call == "adjoint":
        ld, grad, dmu = _Model(par[0], case["dtau"]).logdet_grad()
        return {"logdet": ld, "grad": grad, "dmu": dmu}
    # seconds of the loops below: proposals, and a product over all slices at
    # every interval
    cost = sum(p["Nlx"] * p["Nly"] * p["Ltrot"] * (1.0e-4 + 4.0e-9 * p["Nlx"] * p["Nly"] * p["Ltrot"])
               for p in par)
    if call == "global" or cost > 12.0:
        return None
    models = [_Model(p, case["dtau"]) for p in par]
    done = [m.bin() for m in models]
    out = {"obs": np.stack([obs for obs, _ in done])}
    for i in _read(case):
        m = models[i]
        out["chain%d" % i] = {"sigma": m.sigma.T.astype(np.int8), "seed": m.state, "G": done[i][1]}
    if call == "tau":
        out.update({"tau%d" % i: None for i in range(case["chains"])})
    return out
