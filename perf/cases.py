"""What the speed of this framework is measured on: the passes that a simulation runs over and over.

A pass of most cases is one measurement bin of a batch of Markov chains, as the run-directory driver
takes it: a sweep (left and right traversal of imaginary time), the bin records and the chains' state
back on the host for the checkpoint, and the Green's functions of some chains.  The others are a
restart from a checkpoint, a learned global move with its sweep, a sweep with the time-displaced pass,
and one gradient of the proposer's training.

A case's parameters keep the chains in the phase that simulations of this model run in (no condensate,
mu below the band by a few 1/beta), where every estimator is well above rounding.
"""
from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

import bafqmc_b200
from bafqmc_b200 import workloads
from bafqmc_b200.params import SolverParams
from bafqmc_b200.proposer import Proposer, init_params
from bafqmc_b200.solver import Ensemble

DATA = Path(bafqmc_b200.__file__).resolve().parent / "data"
GREENS = 16         # chains whose Green's function is read after a pass
SITE_SLOT = 32      # first site density of a chain's bin record


def sweep_case(name, lx, ly, L, nwrap, chains, *, dtau=0.05, mu=None, U2=-0.5, delta=0.0, mixed=False):
    beta = dtau * L
    if mu is None:
        mu = max(-7.0, -3.0 - 5.0 / beta)
    return dict(kind="sweep", name=name, lx=lx, ly=ly, L=L, nwrap=nwrap, chains=chains, beta=beta, mu=mu, U1=1.0,
                U2=U2, delta=delta, mixed=mixed)


def listed():
    return [
        # one chain of the smallest cluster: the exact-diagonalisation checks, where only latency counts
        sweep_case("3x3 one chain", 3, 3, 40, 10, 1, dtau=0.1, mu=-4.0, U2=0.0),
        # parameter scans on a small cluster
        sweep_case("4x4 batch", 4, 4, 80, 10, 1500),
        # the benchmark's plain arm: 4096 chains, 160 slices, stabilisation every 10
        sweep_case("6x6 batch", 6, 6, 160, 10, 4096),
        # an odd lattice between the tuned sizes, short stabilisation interval
        sweep_case("7x9 batch", 7, 9, 66, 6, 200),
        # the largest lattice, a chain per SM
        sweep_case("12x12 batch", 12, 12, 50, 10, 148),
        # a restart from a checkpoint in mixed precision: fields in, factors and weights rebuilt (a whole sweep's
        # records in mixed precision carry the rounding of every single-precision product)
        dict(sweep_case("12x12 mixed restart", 12, 12, 100, 10, 148, mixed=True), kind="restart"),
        # the pairing solver on the small and on its largest cluster
        sweep_case("nambu 4x4", 4, 4, 40, 10, 592, mu=-7.0, delta=0.25),
        sweep_case("nambu 6x6", 6, 6, 40, 10, 148, mu=-7.0, delta=0.25),
        # a phase-diagram scan: lattices, temperatures and both sectors in one handle
        dict(kind="ragged", name="ragged grid", per_point=8, mu=-6.0),
        # the learned sampler's step: one network proposal of every chain, accepted exactly, then one sweep
        dict(sweep_case("learned 6x6", 6, 6, 160, 10, 1024), kind="learned"),
        # time-displaced Green's functions in every sweep
        dict(sweep_case("time-displaced 5x7", 5, 7, 60, 6, 148), kind="tau"),
        # one training batch of the proposer: loss and gradient of every parameter
        dict(kind="train", name="train 6x6", lx=6, ly=6, L=160, width=64, batch=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep", "mixed", "nambu", "nambu", "learned", "tau", "train"])
    nwrap = rng.choice([5, 6, 8, 10])
    if kind == "train":
        lx, ly = rng.choice([(3, 4), (4, 4), (4, 5), (6, 6), (4, 7)])
        return dict(kind="train", lx=lx, ly=ly, L=32 * rng.randint(1, 5), width=64, batch=_log_int(rng, 8, 64))
    if kind == "learned":
        lx, ly = rng.choice([(4, 4), (4, 5), (6, 6)])
        c = sweep_case("", lx, ly, 32 * rng.randint(2, 5), 8, _log_int(rng, 64, 1024))
    elif kind == "tau":
        lx, ly = rng.randint(3, 6), rng.randint(3, 6)
        c = sweep_case("", lx, ly, nwrap * rng.randint(4, 8), nwrap, _log_int(rng, 4, 200))
    elif kind == "nambu":
        lx, ly = rng.randint(2, 6), rng.randint(2, 6)
        c = sweep_case("", lx, ly, nwrap * rng.randint(3, 6), nwrap, _log_int(rng, 8, 600 if lx * ly <= 18 else 150),
                       mu=-7.0, delta=rng.choice([0.25, 0.5]))
    else:
        lo, hi = (9, 12) if kind == "mixed" else (3, 12)
        lx, ly = rng.randint(lo, hi), rng.randint(lo, hi)
        big = lx * ly
        cap = 4000 if big <= 16 else (2000 if big <= 36 else (300 if big <= 72 else 148))
        blocks = rng.randint(3, 5) if big > 72 else rng.randint(4, 16)
        c = sweep_case("", lx, ly, nwrap * blocks, nwrap, _log_int(rng, 1, cap), mixed=kind == "mixed")
    c["kind"] = {"mixed": "restart", "nambu": "sweep"}.get(kind, kind)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
def _point(c):
    kw = dict(U1=c["U1"], U2=c["U2"], mu=c["mu"], Nlx=c["lx"], Nly=c["ly"], Ltrot=c["L"], Beta=c["beta"],
              NlxTherm=c["lx"], NlyTherm=c["ly"], LtrotTherm=c["L"], Nwrap=c["nwrap"], Nbin=1, Nsweep=1, iniType=2,
              iniAmpl=1.0)
    if c["delta"]:
        return SolverParams(**kw, shiftLoc=1.0, delta=c["delta"], sector=1)
    return SolverParams(**kw, shiftLoc=1.5)


def _points(c):
    """The case's parameter points and the point of each chain."""
    if c["kind"] != "ragged":
        return [_point(c)], np.zeros(c["chains"], dtype=np.int32)
    pts = [p for p in workloads.ragged_grid() if p.mu == c["mu"] and p.U2 == 0.0]
    return pts, np.repeat(np.arange(len(pts), dtype=np.int32), c["per_point"])


def _start(c, seed):
    """Seeds and N(0,1) fields of every chain, back to back in the order of confin.txt."""
    pts, chain_point = _points(c)
    rng = np.random.default_rng(seed)
    seeds = (2 * rng.integers(1, 2 ** 30 - 1, chain_point.size) + 1).astype(np.int32)
    total = sum(pts[p].Ltrot * pts[p].Lq * 2 for p in chain_point)
    return seeds, rng.standard_normal(total)


def _net_params(width, seed):
    """He-uniform weights with a small random last layer, as a network in training has them."""
    p = init_params(width, seed)
    tail = 27 * 4 * width + 4
    p[-tail:-4] = np.random.default_rng(seed + 1).uniform(-0.01, 0.01, tail - 4).astype(np.float32)
    return p


def _pinned(n, dtype):
    t = torch.empty(n, dtype=dtype, pin_memory=torch.cuda.is_available())
    return t, t.numpy()


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "train":
        rng = np.random.default_rng(seed)
        shape = (c["batch"], c["L"], c["lx"] * c["ly"], 2)
        return dict(kind="train", phi=rng.standard_normal(shape), target=rng.standard_normal(shape),
                    net=Proposer(c["lx"], c["ly"], c["L"], width=c["width"], params=_net_params(c["width"], seed)))
    pts, chain_point = _points(c)
    seeds, phi = _start(c, seed)
    ens = Ensemble(pts, chain_point)
    torch.cuda.synchronize()   # the new handle's memory is cleared on the default stream
    ens.set_state_flat(seeds, phi)
    if c.get("mixed"):
        ens.set_precision("mixed")
    if c["kind"] == "tau":
        ens.set_time_displaced(True, c["L"] // 2 + 1)
    ens.pre()
    ens.synchronize()
    # the host side of a checkpoint: pinned buffers that the state is read into, or a restart from them
    tseeds, nseeds = _pinned(seeds.size, torch.int32)
    tphi, nphi = _pinned(phi.size, torch.float64)
    nseeds[:], nphi[:] = seeds, phi
    state = dict(kind=c["kind"], ens=ens, nseeds=nseeds, nphi=nphi, keep=(tseeds, tphi),
                 greens=range(0, ens.nchains, max(1, ens.nchains // GREENS)))
    if c["kind"] == "learned":
        if (c["lx"], c["ly"], c["L"]) == (6, 6, 160):   # the parameters that ship for this lattice
            state["net"] = Proposer.load(DATA / "proposer_6x6_beta8.npz")
        else:
            state["net"] = Proposer(c["lx"], c["ly"], c["L"], params=init_params(64, 1))
    return state


def run(state):
    if state["kind"] == "train":
        loss, grad = state["net"].loss_grad(state["phi"], state["target"])
        return {"loss": loss, "grad": grad}
    ens = state["ens"]
    if state["kind"] == "restart":
        ens.set_state_flat(state["nseeds"], state["nphi"])
        ens.pre()
        return {"log_weight": ens.log_weight(), "greens": np.stack([ens.green(k) for k in state["greens"]][:GREENS])}
    out = {}
    if state["kind"] == "learned":
        out["accepted"], out["hastings"] = ens.learned_move(state["net"])
    ens.sweep(1)
    out["records"] = ens.chain_obs_raw()
    ens.get_state_flat(state["nseeds"], state["nphi"])
    out["seeds"], out["fields"] = state["nseeds"], state["nphi"]
    if state["kind"] == "ragged":
        out["greens"] = [ens.green(k) for k in state["greens"]][:GREENS]
    else:
        out["greens"] = np.stack([ens.green(k) for k in state["greens"]][:GREENS])
    if state["kind"] == "tau":
        out["displaced"] = np.stack(ens.time_displaced_probe(0))
    return out


def _sweep_work(p, chains):
    n, L, ns = p.block_dim, p.Ltrot, p.Lq
    channels = (abs(p.U1) > 0) + (abs(p.U2) > 0)
    # three complex x real N^3 products a slice and direction, the accepted rank-1 (Nambu: rank-2) updates,
    # pivoted QR, Q and the Green's function at each stabilisation
    acc = 0.85 * 2 * L * ns * channels
    flops = 2 * L * 12.0 * n ** 3 + 8.0 * n ** 2 * acc * (n // ns) + 2.0 * (L // p.Nwrap) * 60.0 * n ** 3
    # fields in and out, G in and out, the stored factors of every stabilisation read and written once a direction
    bytes_ = 2 * 8 * L * ns * 2 + 2 * 16 * n * n + 2 * 2 * (L // p.Nwrap) * 16 * 2 * n * n + 8 * (32 + ns)
    return flops * chains, bytes_ * chains


def work(case):
    c = dict(case)
    if c["kind"] in ("train", "learned"):
        points = c["lx"] * c["ly"] * c["L"]
        w = c.get("width", 64)
        layers = 2.0 * 27 * (2 * w + w * w + w * w + w * 4) * points
        fields = points * 2 * 8
        if c["kind"] == "train":   # forward, the gradients of the weights, and of every layer's input but the first
            return dict(bytes=c["batch"] * 2 * fields + 4 * 27 * (2 * w + 2 * w * w + 4 * w),
                        flops=c["batch"] * (3 * layers - 2.0 * 27 * 2 * w * points))
    if c["kind"] == "ragged":
        pts, _ = _points(c)
        parts = [_sweep_work(p, c["per_point"]) for p in pts]
        return dict(flops=sum(f for f, _ in parts), bytes=sum(b for _, b in parts))
    flops, bytes_ = _sweep_work(_point(c), c["chains"])
    if c["kind"] == "restart":   # one product a slice, one factorisation a stabilisation, one Green's function
        p = _point(c)
        n, Nst = p.block_dim, p.Ltrot // p.Nwrap
        return dict(flops=c["chains"] * n ** 3 * (p.Ltrot * 4.0 + Nst * 24.0 + 60.0),
                    bytes=c["chains"] * (8 * p.Ltrot * p.Lq * 2 + 16 * n * n * (1 + Nst * 2)))
    if c["kind"] == "learned":   # two network passes, and the proposal's factors rebuilt from its fields
        p = _point(c)
        n = p.block_dim
        flops += c["chains"] * (2 * layers + p.Ltrot * 4.0 * n ** 3 + (p.Ltrot // p.Nwrap) * 60.0 * n ** 3)
        bytes_ += c["chains"] * 3 * fields
    if c["kind"] == "tau":       # three functions a slice, and a 2N x 2N inverse a stabilisation
        p = _point(c)
        n = p.block_dim
        flops += c["chains"] * (p.Ltrot * 4 * 4.0 * n ** 3 + (p.Ltrot // p.Nwrap) * (2 * 60.0 * n ** 3 + 30.0 * 8 * n ** 3))
        bytes_ += c["chains"] * (p.Ltrot // p.Nwrap) * 16 * 4 * n * n
    return dict(flops=flops, bytes=bytes_)


# ---------------------------------------------------------------------------
# What a pass returns, from dense 64-bit arithmetic: the same draws and decisions, and G from the whole
# product of slice matrices instead of stabilised factors.
A, MOD = 48828125, 2 ** 31


class _Dense:
    def __init__(self, p, phi, seeds, dev):
        self.p, self.phi, self.seed, self.dev = p, phi, seeds, dev
        ns, self.pair = p.Lq, p.sector == 1
        lx, ly = p.Nlx, p.Nly
        H = np.zeros((p.block_dim, p.block_dim))
        self.bonds = [((x + dx) % lx) + lx * ((y + dy) % ly) for y in range(ly) for x in range(lx)
                      for dx, dy in ((1, 0), (0, 1), (-1, 1))]
        for b, j in enumerate(self.bonds):
            i = b // 3
            for r, s in ((i, j), (j, i)):
                H[r, s] += 1.0
                if self.pair:
                    H[ns + s, ns + r] -= 1.0
        for i in range(ns):
            H[i, i] -= p.mu
            if self.pair:
                H[i, ns + i] += p.delta
                H[ns + i, i] -= p.delta
                H[ns + i, ns + i] += p.mu
        H = torch.tensor(H, dtype=torch.float64, device=dev)
        dtau = p.Beta / p.Ltrot
        z = torch.complex128
        self.expP, self.expM = torch.matrix_exp(-dtau * H).to(z), torch.matrix_exp(dtau * H).to(z)
        self.alpha = [complex(0.0, math.sqrt(2 * p.U1 * dtau)), complex(math.sqrt(-2 * p.U2 * dtau), 0.0)]
        self.active = [ch for ch, u in ((0, p.U1), (1, p.U2)) if abs(u) > 1e-10]
        site = np.arange(ns)
        d = lambda v, m: torch.tensor((v[:, None] - v[None, :]) % m, device=dev)  # noqa: E731
        self.phase = None
        if lx % 3 == 0 and ly % 3 == 0:
            k = 2 * math.pi / 3 * (2 * d(site % lx, lx) + d(site // lx, ly)).double()
            self.phase = torch.complex(k.cos(), k.sin())
        self.obs = torch.zeros(phi.shape[0], SITE_SLOT + ns, dtype=torch.float64, device=dev)

    def factor(self, ch, phi):
        """Diagonal of the HS factor of channel ch for fields [..., ns]."""
        f = torch.exp(self.alpha[ch] * phi)
        if not self.pair:
            return f
        return torch.cat([f, torch.exp((-1.0 if ch == 1 else 1.0) * self.alpha[ch] * phi)], dim=-1)

    def green(self, nt):
        """(I - B)^-1 for the product B of all slices that ends with slice nt."""
        p, n = self.p, self.p.block_dim
        L, C = p.Ltrot, self.phi.shape[0]
        order = [(nt + k) % L for k in range(L)]
        eye = torch.eye(n, dtype=torch.complex128, device=self.dev)
        # a pairing chain's product spans too many decades for one inverse: the block-cyclic matrix of its parts
        parts = L // p.Nwrap if self.pair else 1
        prods = []
        for k in range(parts):
            B = eye.expand(C, n, n)
            for t in order[k * L // parts:(k + 1) * L // parts]:
                v = 1.0
                for ch in self.active:
                    v = v * self.factor(ch, self.phi[:, t, :, ch])
                B = self.expP @ (v[:, :, None] * B)
            prods.append(B)
        if parts == 1:
            return torch.linalg.inv(eye - prods[0])
        M = torch.eye(n * parts, dtype=torch.complex128, device=self.dev).repeat(C, 1, 1)
        for k, B in enumerate(prods):
            r = (k + 1) % parts
            M[:, r * n:(r + 1) * n, k * n:(k + 1) * n] -= B
        rhs = torch.zeros(n * parts, n, dtype=torch.complex128, device=self.dev)
        rhs[:n] = eye
        return torch.linalg.solve(M, rhs.expand(C, -1, -1))[:, :n].contiguous()

    def update(self, G, ch, t, left):
        p, ns = self.p, self.p.Lq
        old = self.phi[:, t, :, ch].clone()
        visit = list(range(ns - 1, -1, -1)) if left else list(range(ns))
        s, u = self.seed, []
        for _ in range(2 * ns):
            s = (s * A) % MOD
            u.append(s.double() / MOD)
        self.seed = s
        f_old = self.factor(ch, old)
        if not left:
            G = G * f_old[:, :, None] / f_old[:, None, :]
        eye = torch.eye(2, dtype=torch.complex128, device=self.dev)
        final = old.clone()
        shift = abs(p.shiftLoc)
        for m, i in enumerate(visit):
            new = old[:, i] + (u[2 * m] - 0.5) * shift
            d = self.factor(ch, (new - old[:, i])[:, None]) - 1.0
            gauss = torch.exp(-0.5 * new ** 2) / torch.exp(-0.5 * old[:, i] ** 2)
            if self.pair:
                idx = [i, ns + i]
                P = eye + d[:, :, None] * (eye - G[:, idx][:, :, idx])
                det = P[:, 0, 0] * P[:, 1, 1] - P[:, 0, 1] * P[:, 1, 0]
                const = torch.exp(self.alpha[ch] * (old[:, i] - new)).abs() if ch == 1 else 1.0
                ok = gauss * const / det.abs() > u[2 * m + 1]
                adj = torch.stack([torch.stack([P[:, 1, 1], -P[:, 0, 1]], 1),
                                   torch.stack([-P[:, 1, 0], P[:, 0, 0]], 1)], 1) / det[:, None, None]
                X = G[:, :, idx] @ (adj * d[:, None, :]) * -ok[:, None, None].double()
                Y = -G[:, idx, :]
                Y[:, 0, i] += 1.0
                Y[:, 1, ns + i] += 1.0
                G = torch.baddbmm(G, X, Y)
            else:
                w = 1.0 + d[:, 0] * (1.0 - G[:, i, i])
                ok = gauss / w.abs() ** 2 > u[2 * m + 1]
                X = G[:, :, i:i + 1] * (-d[:, 0] / w * ok.double())[:, None, None]
                Y = -G[:, i:i + 1, :]
                Y[:, 0, i] += 1.0
                G = torch.baddbmm(G, X, Y)
            final[:, i] = torch.where(ok, new, old[:, i])
        self.phi[:, t, :, ch] = final
        if left:
            f = self.factor(ch, final)
            G = G * f[:, None, :] / f[:, :, None]
        return G

    def measure(self, G):
        p, ns, o = self.p, self.p.Lq, self.obs
        hop = torch.arange(ns, device=self.dev).repeat_interleave(3)
        jj = torch.tensor(self.bonds, device=self.dev)
        eye = torch.eye(ns, dtype=torch.complex128, device=self.dev)
        tr = lambda m: torch.diagonal(m, dim1=1, dim2=2)  # noqa: E731
        if self.pair:
            a, b, c, d = G[:, :ns, :ns], G[:, :ns, ns:], G[:, ns:, :ns], G[:, ns:, ns:]
            nb, nc, gc = -tr(d).conj(), -tr(d), -d
            same = nb[:, :, None] * nb[:, None, :] - d.conj() * a
            cross = nb[:, :, None] * nc[:, None, :] - c.conj() * b
        else:
            gc = G.transpose(1, 2) - eye
            nb = tr(gc)
            same = nb[:, :, None] * nb[:, None, :] + gc * G
            cross = nb[:, :, None] * nb.conj()[:, None, :]
        dens = nb.real.sum(1)
        onsite2 = (nb ** 2).real.sum(1)
        kin = 2.0 * (gc[:, hop, jj] + gc[:, jj, hop]).real.sum(1) / ns
        s_same, s_cross = same.sum((1, 2)), cross.sum((1, 2))
        if self.pair:
            onsite = ((nb * nb + nb * tr(a)).real).sum(1)
            dbl = tr(cross).real.sum(1) / ns
            pairing = (tr(c) - tr(b)).real.sum(1) / ns
        else:
            onsite = 2.0 * onsite2 + dens
            dbl = (nb.abs() ** 2).sum(1) / ns
        inter = (p.U1 + p.U2) * 2.0 * onsite / ns + 2.0 * (p.U2 - p.U1) * dbl
        energy = kin + inter
        o[:, 0] += dens / ns
        o[:, 1] += dens / ns
        o[:, 2] += 2.0 * dens / ns
        o[:, 3] += kin
        o[:, 4] += dbl
        o[:, 5] += 2.0 * onsite2 / ns
        o[:, 6] += dens
        o[:, 7] += dens
        o[:, 8] += s_same.real
        o[:, 9] += s_same.real
        o[:, 10] += onsite
        o[:, 11] += onsite
        o[:, 12] += inter
        if self.pair:
            energy = energy + p.delta * pairing
            o[:, 26] += 2.0 * dens / ns
            o[:, 27] += 2.0 * onsite / ns
            o[:, 28] += pairing
            o[:, 29] += p.delta * pairing
            o[:, 30] += -p.mu * 2.0 * dens / ns
            o[:, 31] += energy - p.mu * 2.0 * dens / ns
            bc = tr(c).sum(1) * tr(b).sum(1)
            o[:, 16] += ((d.abs() ** 2).sum((1, 2)) - bc.real) / ns ** 2
            o[:, 17] += bc.imag / ns ** 2
        else:
            o[:, 16] += (gc.abs() ** 2).sum((1, 2)) / ns ** 2
        o[:, 13] += energy
        if self.phase is not None:
            sf = (self.phase * 2.0 * gc.real).sum((1, 2)) / ns ** 2
            dw = (self.phase * 2.0 * (same + cross).real).sum((1, 2)) / ns ** 2
            for k, v in ((14, sf), (18, dw)):
                o[:, k] += v.real
                o[:, k + 1] += v.imag
        for k, v in ((20, s_same), (22, s_same.conj()), (24, s_cross)):
            o[:, k] += v.real / ns
            o[:, k + 1] += v.imag / ns
        o[:, SITE_SLOT:] += 2.0 * nb.real

    def sweep(self):
        L, W = self.p.Ltrot, self.p.Nwrap
        for nt in range(L, 0, -1):
            if nt % W == 0:
                G = self.green(nt)
            self.measure(G)
            G = self.expM @ G @ self.expP
            for ch in reversed(self.active):
                G = self.update(G, ch, nt - 1, True)
        G = self.green(0)
        for nt in range(1, L + 1):
            for ch in self.active:
                G = self.update(G, ch, nt - 1, False)
            G = self.expP @ G @ self.expM
            if nt % W == 0:
                G = self.green(nt)
            self.measure(G)
        self.obs /= 2 * L
        return G


def _dense_gradient(c, seed):
    """Loss and gradient of the network in float64 (its bf16 weights, no rounding between layers)."""
    s = prepare(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    w, out = c["width"], []
    flat = torch.tensor(_net_params(w, seed), dtype=torch.float64, device=dev).requires_grad_()
    B, L, ns, _ = s["phi"].shape
    grid = lambda v: torch.tensor(v, device=dev).reshape(B, L, c["ly"], c["lx"], 2).permute(0, 4, 1, 2, 3)  # noqa: E731
    x = grid(s["phi"]).to(torch.bfloat16).double()
    at = 0
    for l, (ci, co) in enumerate([(2, w), (w, w), (w, w), (w, 4)]):
        k = flat[at:at + 27 * ci * co].reshape(3, 3, 3, co, ci)   # offsets (y, x, t)
        at += 27 * ci * co
        bias = flat[at:at + co]
        at += co
        k = k + (k.detach().to(torch.bfloat16).double() - k.detach())
        y = 0.0
        for b in range(3):
            for cc in range(3):
                for a in range(3):
                    moved = torch.roll(x, shifts=(1 - a, 1 - b, 1 - cc), dims=(2, 3, 4))
                    y = y + torch.einsum("oi,nityx->notyx", k[b, cc, a], moved)
        x = y + bias[None, :, None, None, None]
        if l < 3:
            x = torch.relu(x)
    z = (grid(s["target"]) - x[:, :2]) * torch.exp(-x[:, 2:])
    loss = (0.5 * z * z + x[:, 2:]).mean()
    loss.backward()
    return {"loss": float(loss), "grad": flat.grad.cpu().numpy()}


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "train":
        return _dense_gradient(c, seed) if c["batch"] * c["lx"] * c["ly"] * c["L"] <= 400000 else None
    if c["kind"] in ("ragged", "learned"):
        return None    # a bf16 network decides, or many points one after another: minutes of dense arithmetic
    p = _point(c)
    # a sequential visit of every site, slice and channel, each a few passes over all chains' matrices
    visits = 2 * p.Ltrot * p.Lq * 2
    if c["kind"] != "restart" and visits * (3e-4 + 3e-12 * c["chains"] * 16 * p.block_dim ** 2) > 16.0:
        return None
    if c["delta"] and p.block_dim * p.Ltrot // p.Nwrap > 400:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    seeds, phi = _start(c, seed)
    phi = torch.tensor(phi.reshape(c["chains"], p.Ltrot, p.Lq, 2), device=dev)
    d = _Dense(p, phi, torch.tensor(seeds.astype(np.int64), device=dev), dev)
    some = list(range(0, c["chains"], max(1, c["chains"] // GREENS)))[:GREENS]
    if c["kind"] == "restart":
        G = d.green(p.Ltrot)
        weight = -0.5 * (phi ** 2).sum((1, 2, 3)) + 2.0 * torch.linalg.slogdet(G)[1]
        return dict(log_weight=weight.cpu().numpy(), greens=G[some].cpu().numpy())
    G = d.sweep()
    out = dict(records=d.obs.cpu().numpy(), seeds=None, fields=d.phi.reshape(-1).cpu().numpy(),
               greens=G[some].cpu().numpy())
    if c["kind"] == "tau":
        out["displaced"] = None
    return out
