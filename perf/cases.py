"""Performance cases: what users of the framework run, through its public entry points.

The unit of work is what a driver program does between two measurements: a few graph
substeps of the walker set on the device, then the energy, then the walker records read
back.  The listed cases are the sizes of the workload table (`synthetic.CONFIGS`,
`synthetic.C5_SYSTEMS`), in the numerical form each is run in, one odd-sized system in
each form with complex orbitals and Cholesky vectors, and the calls a program makes on
their own (an exact measurement, a restart from host memory, the exchange energy of
another framework's buffers).

A case's Hamiltonian is that of its sizes (a fixed synthetic molecule, as a run keeps one
Hamiltonian); the seed makes the walkers, their weights and the auxiliary fields.  Every
pass starts from the same walkers: they are kept in a second walker set and copied on the
device, so that a pass can be repeated without the trajectory running away.

The mixed form computes to about single precision (split bf16 operands, fp32 sums), and a
program that runs it keeps its results in single precision, as `run` does here; the FP64
form's results stay in double precision.
"""
from __future__ import annotations

import ctypes
import math
from types import SimpleNamespace

import numpy as np
import torch

from miniafqmc_b200 import afqmc
from miniafqmc_b200.synthetic import CSR, HALFROTATE_CUTOFF, Config, System

ORDER, NORTHO = 6, 5


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest run: a 64-orbital system, 16 walkers, energy after every step with
        # the stored two-body matrix; launches and latency count
        _c("small_fp64_run", "interval", "fp64", 64, 16, 256, 0.10, 16, steps=20, every=1,
           energy="vakbl", walkers_out=True),
        # the same system in the mixed form, as a first try or an interactive session runs it
        _c("small_mixed_interval", "interval", "mixed", 64, 16, 256, 0.10, 16, steps=5),
        # an ordinary production set in full double precision, energy every 2 substeps
        _c("medium_fp64_interval", "interval", "fp64", 128, 32, 512, 0.05, 256, steps=2),
        # odd sizes, complex orbitals and Cholesky vectors, operations called one by one
        # with the fields of the caller's own generator
        _c("ragged_fp64_stages", "stages", "fp64", 77, 13, 301, 0.25, 53, steps=3, cplx=True,
           walkers_out=True),
        # walkers, electrons and columns that fill no tile, in the mixed form (whose operand
        # rows are multiples of 16 bytes: orbitals and Cholesky vectors in eights, electrons
        # in fours)
        _c("ragged_mixed_interval", "interval", "mixed", 184, 28, 616, 0.15, 131, steps=5,
           cplx=True),
        # dense Cholesky vectors and 64+64 electrons, mixed form, exact energies
        _c("dense_mixed_interval", "interval", "mixed", 256, 64, 1024, 0.30, 512, steps=5),
        # the largest system in double precision: the reference run that others are checked
        # against
        _c("large_fp64_interval", "interval", "fp64", 384, 48, 1536, 0.20, 128, steps=2),
        # the same system in the form long runs use: mixed, 1024 walkers, energies with the
        # learned control variate every 5 substeps
        _c("large_mixed_cv_interval", "interval", "mixed", 384, 48, 1536, 0.20, 1024, steps=5,
           energy="cv"),
        # an exact measurement of such walkers on its own (density matrix and energy)
        _c("large_mixed_measure", "measure", "mixed", 384, 48, 1536, 0.20, 512),
        # three systems of uneven size advanced together, energies after 5 substeps
        _c("batch_mixed_interval", "batch", "mixed", 0, 0, 0, 0.10, 0, steps=5),
        # a restarted job: walkers from host memory, 10 substeps, walkers back to the host
        _c("restart_mixed", "restart", "mixed", 200, 40, 800, 0.10, 256, steps=10,
           walkers_out=True),
        # exchange energies of density matrices that another framework's pool holds
        _c("exchange_of_buffers", "exchange", "fp64", 200, 40, 800, 0.10, 96, cplx=True),
    ]


def _c(name, kind, form, nmo, nel, nchol, density, nwalk, steps=0, every=0, energy="chol",
       cplx=False, walkers_out=False):
    c = dict(kind=kind, form=form, nmo=nmo, nel=nel, nchol=nchol, density=density, nwalk=nwalk,
             steps=steps, every=every or steps, energy=energy, cplx=cplx,
             walkers_out=walkers_out)
    return dict(c, name=name) if name else c


def draw(rng):
    """A case of the same ranges: 48 to 384 orbitals (odd numbers among them), 4 to 64
    electrons of each spin, 2 to 4 Cholesky vectors per orbital, 5% to 30% nonzero, 8 to
    1024 walkers (fewer where the case would cost more than the largest listed one)."""
    top = {"fp64": work(listed()[6]), "mixed": work(listed()[7])}
    while True:
        form = rng.choice(["fp64", "mixed"])
        kind = rng.choice(["interval", "interval", "interval", "stages", "measure", "restart",
                           "exchange"])
        nmo = round(math.exp(rng.uniform(math.log(48), math.log(384))))
        nel = rng.randint(4, min(64, nmo // 3))
        nchol = round(nmo * rng.uniform(2.0, 4.0))
        nwalk = round(math.exp(rng.uniform(math.log(8), math.log(1024))))
        if form == "mixed" and kind != "exchange":   # operand rows of whole 16 bytes
            nmo, nel, nchol = nmo // 8 * 8, max(4, nel // 4 * 4), nchol // 8 * 8
        if kind == "exchange":
            form = "fp64"
            nwalk = min(nwalk, (1 << 17) // math.ceil(nchol / (96 // nel)))
        if kind == "restart":
            nwalk = min(nwalk, 256)
        c = _c("", kind, form, nmo, nel, nchol, round(rng.uniform(0.05, 0.30), 3), nwalk,
               steps=0 if kind in ("measure", "exchange") else rng.randint(1, 5),
               cplx=rng.random() < 0.3, walkers_out=kind == "restart")
        w = work(c)
        if w["flops"] <= 0.5 * top[form]["flops"] and w["bytes"] <= 0.5 * top["mixed"]["bytes"]:
            return c


# ------------------------------------------------------------------ Hamiltonians
_SYSTEMS: dict = {}   # the Hamiltonians of the case in hand, by sizes


def _shapes(case):
    """(nmo, nel, nchol, density, nwalk) of the case's systems."""
    if case["kind"] == "batch":
        return [(96, 12, 384, 0.10, 128), (200, 40, 800, 0.10, 256), (320, 64, 1280, 0.10, 384)]
    return [(case["nmo"], case["nel"], case["nchol"], case["density"], case["nwalk"])]


def _systems(case):
    keys = [s[:4] + (case["cplx"], case["energy"] == "vakbl") for s in _shapes(case)]
    if any(k not in _SYSTEMS for k in keys):
        _SYSTEMS.clear()
        for k in keys:
            _SYSTEMS[k] = _make_system(*k)
    return [_SYSTEMS[k] for k in keys]


def _gen(*key):
    """A torch generator on the GPU for this key."""
    seed = 0
    for k in key:
        seed = (seed * 1000003 + int(k)) % (1 << 62)
    return torch.Generator("cuda").manual_seed(seed)


def _randn(g, *shape, cplx=False):
    x = torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)
    if cplx:
        x = torch.complex(x, torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64))
    return x


def _csr(dense) -> CSR:
    """CSR of a dense device matrix."""
    mask = dense != 0
    ri = torch.zeros(dense.shape[0] + 1, dtype=torch.int64, device="cuda")
    ri[1:] = mask.sum(1).cumsum(0)
    cols = mask.nonzero()[:, 1].to(torch.int32).cpu().numpy()
    vals = dense[mask].to(torch.complex128).cpu().numpy()
    return CSR(dense.shape[0], dense.shape[1], ri.to(torch.int32).cpu().numpy(), cols, vals)


def _make_system(N, n, nchol, density, cplx, vakbl) -> System:
    """The synthetic molecule of `miniafqmc_b200.synthetic` for these sizes, made on the GPU:
    one-body matrix with a spread diagonal, symmetric sparse Cholesky vectors, the lowest
    eigenvectors as the trial, the one-body propagator and the half-rotated factors."""
    cfg = Config(N, n, nchol, density, 0, taylor_order=ORDER)
    g = _gen(17, N, n, nchol, round(1000 * density), cplx)
    A = 0.1 * _randn(g, N, N)
    h1 = 0.5 * (A + A.T) + torch.diag(torch.linspace(-2, 2, N, device="cuda", dtype=torch.float64))
    keep = torch.rand(nchol, N, N, generator=g, device="cuda") < density
    L = torch.where(keep, cfg.sigma * _randn(g, nchol, N, N), 0.0).triu()
    if cplx:
        L = torch.complex(L, torch.where(keep, 0.4 * cfg.sigma * _randn(g, nchol, N, N), 0.0).triu())
    del keep
    L = L + L.triu(1).transpose(1, 2)
    wf = torch.linalg.eigh(h1)[1][:, :n].to(torch.complex128)
    if cplx:
        wf = wf @ torch.linalg.qr(_randn(g, n, n, cplx=True))[0]
    trial = torch.stack([wf, wf]).conj().resolve_conj()
    LL = torch.zeros(N, N, dtype=L.dtype, device="cuda")
    for c in range(0, nchol, 64):
        M = L[c:c + 64].transpose(0, 1).reshape(N, -1)
        LL += M @ M.T
    P = torch.linalg.matrix_exp(-0.5 * cfg.dt * (h1.to(LL.dtype) - 0.5 * LL)).to(torch.complex128)
    Lh = torch.empty(nchol, 2, n, N, dtype=torch.complex128, device="cuda")
    for c in range(0, nchol, 64):   # Lh[c][s][a][k] = sum_i trial_s(i, a) L_c(i, k)
        for s in range(2):
            Lh[c:c + 64, s] = trial[s].T @ L[c:c + 64].to(torch.complex128)
    sq = math.sqrt(cfg.dt)
    Ls = Lh.reshape(nchol, -1) * sq
    Ls[Ls.abs() <= HALFROTATE_CUTOFF] = 0.0
    V = None
    if vakbl:
        F = Lh.reshape(nchol, -1)
        J = F.T @ F
        m = n * N
        for s in range(2):
            sl = slice(s * m, (s + 1) * m)
            X = J[sl, sl].reshape(n, N, n, N).permute(0, 3, 2, 1).reshape(m, m).clone()
            J[sl, sl] -= X
        V = _csr(J)
    h1c = h1.to(torch.complex128)
    s = System(cfg=cfg, h1=h1.cpu().numpy(), Wavefun=trial.conj().resolve_conj().cpu().numpy(),
               spvn_coo=(), Propg1=P.cpu().numpy())
    s.Spvn = _csr((L * sq).permute(1, 2, 0).reshape(N * N, nchol))
    s.SpvnT = _csr(Ls)
    s.trial = trial.cpu().numpy()
    s.haj = torch.cat([trial[0].T @ h1c, trial[1].T @ h1c]).cpu().numpy()
    s.Lh = Lh.cpu().numpy()
    s.Vakbl = V
    return s


# ------------------------------------------------------------------ walkers and fields
def _walkers(system, nwalk, seed, spread=0.35):
    """Orthonormal walkers around the trial, as a run has them after some substeps, and
    their records: weights between 0.5 and 1.5."""
    N, n = system.N, system.n
    g = _gen(29, seed, N, n, nwalk)
    ref = torch.from_numpy(np.conj(system.trial)).cuda()
    W = ref + spread / math.sqrt(2 * N) * _randn(g, nwalk, 2, N, n, cplx=True)
    for _ in range(2):
        R = torch.linalg.cholesky(W.mH @ W).mH
        W = torch.linalg.solve_triangular(R, W, upper=True, left=False)
    Wd = np.zeros((nwalk, 8), np.complex128)
    Wd[:, 1] = (0.5 + torch.rand(nwalk, generator=g, device="cuda", dtype=torch.float64)).cpu().numpy()
    return W.contiguous(), Wd


def _fields(case, seed, k):
    return _randn(_gen(31, seed, k), case["nchol"], case["nwalk"])


class _WalkerStore:
    """A second walker set on the device, which passes start from."""

    def __init__(self, system, nwalk, W, Wd):
        self.lib = afqmc.load_library()
        desc = afqmc.SystemDesc(system.N, system.n, system.n, 1, nwalk, system.cfg.dt, ORDER,
                                afqmc.AFQ_PREC_FP64, 0)
        self.h = ctypes.c_void_p()
        st = self.lib.afq_create(ctypes.byref(desc), ctypes.byref(self.h))
        if st == 0:
            st = self.lib.afq_set_walkers(self.h, W.ctypes.data, Wd.ctypes.data)
        if st != 0:
            raise afqmc.AfqmcError(st, "walker store")

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.afq_destroy(self.h)
            self.h = None


def prepare(case, seed):
    systems = _systems(case)
    if case["kind"] == "exchange":
        s, nw = systems[0], case["nwalk"]
        W, _ = _walkers(s, nw, seed)
        st = SimpleNamespace(case=case, Lh=torch.from_numpy(s.Lh).cuda(),
                             G=_density(W, torch.from_numpy(s.trial).cuda())[0].contiguous(),
                             ek=torch.empty(nw, dtype=torch.complex128, device="cuda"))
        return st
    prec = afqmc.AFQ_PREC_FP64 if case["form"] == "fp64" else afqmc.AFQ_PREC_MIXED
    st = SimpleNamespace(case=case, seed=1000 + int(seed), engines=[], stores=[], x=[])
    for s, shape in zip(systems, _shapes(case)):
        Wt, Wd = _walkers(s, shape[4], seed)
        W = Wt.cpu().numpy()
        vak = case["energy"] == "vakbl"
        e = afqmc.AfqmcSys(s, shape[4], precision=prec, use_vakbl=vak, use_chol=not vak,
                           walkers=(W, Wd))
        st.engines.append(e)
        if case["kind"] == "restart":
            st.host = (W, Wd)
        else:
            st.stores.append(_WalkerStore(s, shape[4], W, Wd))
    if case["kind"] == "stages":
        st.x = [_fields(case, seed, k).cpu().numpy() for k in range(case["steps"])]
    if case["kind"] == "batch":
        st.batch = afqmc.AfqmcBatch(st.engines)
    if case["energy"] == "cv":   # a run in progress: the first exact samples are behind it
        st.engines[0].cv_configure()
        for _ in range(3):
            run(st)
    return st


def _result(case, e, energies):
    """The walker records (and the walkers where the program keeps them) of one engine."""
    W = None
    if case["walkers_out"]:
        W, d = e.get_walkers()
    else:
        d = e.get_walker_data()
    out = {"energies": np.array(energies), "local_energy": d[:, 0], "weight": d[:, 1],
           "overlap": d[:, 2:4], "hybrid_energy": d[:, 4:6], "old_overlap": d[:, 6:8]}
    if W is not None:
        out["walkers"] = W
    if case["form"] == "mixed":
        out = {k: v.astype(np.complex64 if np.iscomplexobj(v) else np.float32)
               for k, v in out.items()}
    return out


def run(st):
    case = st.case
    kind = case["kind"]
    if kind == "exchange":
        lib = afqmc.load_library()
        status = lib.afq_exchange_energy_noalloc(
            st.Lh.data_ptr(), st.G.data_ptr(), case["nmo"], case["nel"], case["nchol"],
            case["nwalk"], st.ek.data_ptr(), torch.cuda.current_stream().cuda_stream)
        if status != 0:
            raise afqmc.AfqmcError(status, "exchange energy")
        return st.ek
    e = st.engines[0]
    if kind == "restart":
        e.set_walkers(*st.host)
    else:
        for eng, store in zip(st.engines, st.stores):
            eng.copy_walkers_from(store)
    for eng in st.engines:
        eng.eshift = 0.0
    energies = []
    if kind == "batch":
        st.batch.substeps([st.seed] * len(st.engines), 1, case["steps"], NORTHO)
        out = []
        for eng in st.engines:
            eng.calculate_mixed_density_matrix()
            out.append(_result(case, eng, [eng.calculate_energy(case["energy"])]))
        return out
    if kind == "stages":
        for k, x in enumerate(st.x):
            e.calculate_mixed_density_matrix()
            e.get_vbias()
            e.sigma_from(x)
            e.get_vHS()
            e.propagate()
            e.calculate_overlaps(save_old=True)
            e.update_weights()
        e.orthogonalize()
        e.calculate_overlaps(save_old=False)
    else:
        for k in range(1, case["steps"] + 1):
            e.substep(st.seed, k, NORTHO)
            if k % case["every"] == 0 and k < case["steps"]:
                e.calculate_mixed_density_matrix()
                energies.append(e.calculate_energy(case["energy"]))
    e.calculate_mixed_density_matrix()
    energies.append(e.calculate_energy(case["energy"]))
    return _result(case, e, energies)


# ------------------------------------------------------------------ work
def work(case):
    """Multiply-adds and bytes of one pass: every sparse operand's nonzeros once per
    product, real operands at half the cost of complex ones, the Hamiltonian and the
    walkers read once, the walkers and their records written once."""
    flops = bytes_ = 0.0
    f = 8.0 if case["cplx"] else 4.0          # a Hamiltonian value times a complex number
    hb = 16.0 if case["cplx"] else 8.0
    for N, n, nc, d, nw in _shapes(case):
        nak, walker = 2.0 * n * N, 32.0 * n * N
        exch = f * 2 * nc * float(n) * n * N + 8.0 * nc * n * n * 2
        if case["kind"] == "exchange":
            flops += nw * exch
            bytes_ += 16.0 * nc * nak + 16.0 * nw * nak + 16.0 * nw
            continue
        dm = 8.0 * 2 * N * n * n * 2 + 8.0 * 2 * n ** 3
        sub = dm + f * nc * nak + f * nc * d * N * (N + 1) / 2
        sub += 2 * f * N * nak + ORDER * 8.0 * N * nak                       # the propagation
        sub += 8.0 * 2 * N * n * n + 8.0 * 2 * n ** 3 / 3                    # new overlaps
        meas = dm + 8.0 * nak
        if case["energy"] == "vakbl":
            meas += f * nak * nak
            bytes_ += hb * nak * nak
        else:
            meas += f * nc * nak + exch * (0.125 if case["energy"] == "cv" else 1.0)
            bytes_ += hb * nc * nak
        northo = 1 if case["kind"] == "stages" else case["steps"] // NORTHO
        nmeas = case["steps"] // case["every"] if case["steps"] else 1
        flops += nw * (case["steps"] * sub + nmeas * meas
                       + northo * (8.0 * 4 * N * n * n + 8.0 * 2 * N * n * n))
        bytes_ += nw * (2 * walker + 2 * 128.0)
        if case["steps"]:
            bytes_ += hb * nc * nak + hb * d * nc * N * (N + 1) / 2 + hb * N * N
        if case["kind"] == "stages":
            bytes_ += 8.0 * nc * nw * case["steps"]
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------ 64-bit values
def _density(W, trial):
    """Gc [nw][2][n][N] and the overlaps [nw][2] of walkers [nw][2][N][n]."""
    T1 = W.transpose(2, 3) @ trial
    return torch.linalg.solve(T1, W.transpose(2, 3)), torch.linalg.det(T1)


def _normals(seed, step, count):
    """The first `count` standard normals of the framework's field stream: Philox4x32-10
    (Salmon et al., SC'11) counters (pair, step), key seed, Box-Muller on two 53-bit
    uniforms."""
    pairs = np.arange((count + 1) // 2, dtype=np.uint64)
    lo32 = np.uint64(0xFFFFFFFF)
    c = [pairs & lo32, pairs >> np.uint64(32),
         np.full_like(pairs, step & 0xFFFFFFFF), np.full_like(pairs, step >> 32)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & lo32,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & lo32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = [((a >> np.uint64(5)) << np.uint64(26) | (b >> np.uint64(6))).astype(np.float64)
         for a, b in ((c[0], c[1]), (c[2], c[3]))]
    u1, u2 = (u[0] + 1.0) / 2.0 ** 53, u[1] / 2.0 ** 53
    r, th = np.sqrt(-2.0 * np.log(u1)), 2.0 * np.pi * u2
    return np.stack([r * np.cos(th), r * np.sin(th)], 1).reshape(-1)[:count]


def _dense(csr):
    m = torch.sparse_csr_tensor(torch.from_numpy(csr.rowIndex), torch.from_numpy(csr.cols),
                                torch.from_numpy(csr.vals), (csr.nrows, csr.ncols))
    return m.cuda().to_dense()


class _Exact:
    """One system's trajectory in complex128 matrix products."""

    def __init__(self, case, system, nwalk, seed):
        self.case, self.s, self.nw = case, system, nwalk
        self.W, Wd = _walkers(system, nwalk, seed)
        self.Wd = torch.from_numpy(Wd).cuda()
        cuda = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
        self.trial, self.P, self.haj = cuda(system.trial), cuda(system.Propg1), cuda(system.haj)
        self.Lh = cuda(system.Lh)
        self.eshift = 0.0
        if case["steps"]:
            self.Spvn, self.SpvnT = _dense(system.Spvn), _dense(system.SpvnT)

    def overlaps(self):
        self.Wd[:, 2:4] = _density(self.W, self.trial)[1]

    def substep(self, x):
        s, nw, dt = self.s, self.nw, self.s.cfg.dt
        N, n = s.N, s.n
        G, det = _density(self.W, self.trial)
        self.Wd[:, 2:4] = det
        vb = self.SpvnT @ G.reshape(nw, -1).T
        hw = -(1j * vb * (x + 0.5j * vb)).sum(0)
        X = x + 1j * vb
        S = (self.P @ self.W).transpose(1, 2).reshape(nw, N, 2 * n)
        step = max(1, (1 << 28) // (N * N))
        for w in range(0, nw, step):
            V = (self.Spvn @ X[:, w:w + step]).T.reshape(-1, N, N)
            T = S[w:w + step].clone()
            acc = T.clone()
            for k in range(1, ORDER + 1):
                T = (1j / k) * (V @ T)
                acc += T
            S[w:w + step] = self.P @ acc
        self.W = S.reshape(nw, N, 2, n).transpose(1, 2).contiguous()
        d = self.Wd
        d[:, 5] = d[:, 4]
        d[:, 6:8] = d[:, 2:4]
        self.overlaps()
        ratio = d[:, 2] * d[:, 3] / (d[:, 6] * d[:, 7])
        e4 = -(hw + torch.log(ratio)) / dt
        f = torch.cos(ratio.angle()).clamp(min=0) * torch.exp(
            -dt * (0.5 * (e4.real + d[:, 5].real) - self.eshift))
        d[:, 4] = e4
        d[:, 1] *= f
        self.eshift = float(e4.real.mean())

    def orthogonalize(self):
        if self.case["form"] == "fp64":   # LAPACK's Householder signs
            self.W = torch.linalg.qr(self.W.conj())[0].conj().resolve_conj()
        else:                             # positive diagonal of R
            for _ in range(2):
                R = torch.linalg.cholesky(self.W.mH @ self.W).mH
                self.W = torch.linalg.solve_triangular(R, self.W, upper=True, left=False)
        self.overlaps()

    def energy(self):
        G, det = _density(self.W, self.trial)
        self.Wd[:, 2:4] = det
        e = (G.reshape(self.nw, -1) * self.haj.reshape(-1)).sum(1)
        F = self.Lh.reshape(self.s.nchol, -1)
        cv = F @ G.reshape(self.nw, -1).T
        e = e + 0.5 * (cv * cv).sum(0) - _exchange(self.Lh, G)
        self.Wd[:, 0] = e
        w = self.Wd[:, 1].real
        return float((e.real * w).sum() / w.sum())

    def result(self, energies):
        d = self.Wd
        out = {"energies": torch.tensor(energies, dtype=torch.float64), "local_energy": d[:, 0],
               "weight": d[:, 1], "overlap": d[:, 2:4], "hybrid_energy": d[:, 4:6],
               "old_overlap": d[:, 6:8]}
        if self.case["walkers_out"]:
            out["walkers"] = self.W
        if self.case["energy"] == "cv":   # an estimate: of the surrogate and a random subset
            out["energies"] = out["local_energy"] = None
        return out


def _exchange(Lh, G):
    """1/2 sum_{s,c} tr(T T), T = Lh_s[c] Gc_s^T, of every walker."""
    nc, _, n, N = Lh.shape
    nw = G.shape[0]
    ek = torch.zeros(nw, dtype=torch.complex128, device="cuda")
    real = bool((Lh.imag == 0).all())
    step = max(1, (1 << 27) // (nw * n * n))
    for s in range(2):
        g = G[:, s].reshape(nw * n, N).T.contiguous()
        for c in range(0, nc, step):
            A = Lh[c:c + step, s].reshape(-1, N)
            if real:
                A = A.real.contiguous()
                T = torch.complex(A @ g.real, A @ g.imag)
            else:
                T = A @ g
            T = T.reshape(-1, n, nw, n)
            ek += 0.5 * (T * T.transpose(1, 3)).sum((0, 1, 3))
    return ek


def exact(case, seed):
    if case["kind"] == "exchange":
        s = _systems(case)[0]
        W, _ = _walkers(s, case["nwalk"], seed)
        G, _ = _density(W, torch.from_numpy(s.trial).cuda())
        return _exchange(torch.from_numpy(s.Lh).cuda(), G)
    outs = []
    for system, shape in zip(_systems(case), _shapes(case)):
        nw = shape[4]
        t = _Exact(case, system, nw, seed)
        energies = []
        for k in range(case["steps"]):
            if case["kind"] == "stages":
                x = _fields(case, seed, k)
            else:
                x = torch.from_numpy(_normals(1000 + int(seed), k + 1, system.nchol * nw)
                                     .reshape(system.nchol, nw)).cuda()
            t.substep(x)
            if case["kind"] != "stages":
                if (k + 1) % NORTHO == 0:
                    t.orthogonalize()
                if (k + 1) % case["every"] == 0 and k + 1 < case["steps"]:
                    energies.append(t.energy())
        if case["kind"] == "stages":
            t.orthogonalize()
        if case["energy"] == "cv":
            t.overlaps()
        else:
            energies.append(t.energy())
        outs.append(t.result(energies))
        del t
    return outs if case["kind"] == "batch" else outs[0]
