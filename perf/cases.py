"""What a user of the framework has it do, as measurable cases.

Every case is one call (or one chain of calls) through the package's public
entry points on a clamped Hexa8 block, over the sizes of the configurations,
tests and benchmark of this repository: from the 10 x 4 x 4 cantilever to the
64^3 block, from a handful of realizations to the 1024 of the Monte Carlo
batch, even sides (which the multigrid levels halve) and odd ones.

kinds
  static   StaticAnalyzer -> LinearAnalyzer -> SolverPCG: assembly of the global
           stiffness for the elements' moduli and one PCG solve (FP64 or mixed)
  mc       one Monte Carlo batch, KL field to displacements, inputs and outputs
           on the device, on a cube lattice or on one with moved nodes
  newmark  implicit dynamics of a batch of realizations (host buffers)
  stress   stress recovery of every element of every realization on the device
  galerkin one product with the polynomial-chaos Galerkin operator (host buffers)
  ragged   one Monte Carlo batch over systems of uneven size (host buffers)

Outputs are displacements, strains, stresses and forces. Iteration counts and
final residuals are diagnostics of the loop (they hang on the last bits of its
FP32 arithmetic) and are not returned.
"""
import ctypes
import math

import numpy as np
import torch

import msolve_b200 as M

NU = 0.3
TERMS = 50        # KL terms of the Monte Carlo configurations
MAX_IT = 20000
TOL_MC = 1e-10    # FP64 true residual of a realization: displacements to better than 1e-9 on every block here
TOL_STATIC = 1e-10
TOL_STEP = 1e-13  # Newmark steps (the benchmark's default)


def listed():
    return [
        # the cantilever of the first configuration: one small solve, all latency
        dict(name="static_10x4x4", kind="static", nx=10, ny=4, nz=4, precision="fp64"),
        # an ordinary block of uneven sides, FP32 values with FP64 refinement
        dict(name="static_mixed_37x22x29", kind="static", nx=37, ny=22, nz=29, precision="mixed"),
        # the largest single solve of the configurations
        dict(name="static_64", kind="static", nx=64, ny=64, nz=64, precision="fp64"),
        # a small model's batch, as a serving lane of the smallest model runs it
        dict(name="mc_8_R64", kind="mc", nx=8, ny=8, nz=8, R=64, moved=False),
        # odd sides
        dict(name="mc_21x13x9_R100", kind="mc", nx=21, ny=13, nz=9, R=100, moved=False),
        # an ordinary batch
        dict(name="mc_24_R256", kind="mc", nx=24, ny=24, nz=24, R=256, moved=False),
        # the Monte Carlo configuration
        dict(name="mc_32_R1024", kind="mc", nx=32, ny=32, nz=32, R=1024, moved=False),
        # a block with moved nodes: not a cube lattice
        dict(name="mc_moved_24_R200", kind="mc", nx=24, ny=24, nz=24, R=200, moved=True),
        # dynamics of a batch, ten of the configuration's steps
        dict(name="newmark_24_R256", kind="newmark", n=24, R=256, steps=10),
        # stresses of a batch's realizations
        dict(name="stress_20_R64", kind="stress", n=20, R=64, moved=False),
        # the Galerkin operator of four germs up to degree three (35 blocks)
        dict(name="galerkin_12_m4_p3", kind="galerkin", n=12, m=4, p=3),
        # blocks of uneven size in one call, cube lattices and moved nodes
        dict(name="ragged_8_16_24", kind="ragged", n1=8, n2=16, n3=24, n4=12, n5=20, R=64),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["static", "static", "mc", "mc", "mc", "newmark", "stress", "galerkin", "ragged"])
    if kind == "static":
        return dict(kind=kind, nx=log_int(6, 64), ny=log_int(4, 56), nz=log_int(4, 56),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "mc":
        moved = rng.random() < 0.3
        nx = log_int(6, 40)
        ny, nz = (log_int(max(4, nx // 2), min(32, 3 * nx // 2)) for _ in range(2))
        if rng.random() < 0.5:
            nx = ny = nz = rng.choice([8, 10, 12, 15, 16, 18, 20, 24, 25, 28, 32])
        # no more than a fifth of the Monte Carlo configuration's elements x realizations
        most = max(1, int(6.0e6 / (nx * ny * nz)))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, R=log_int(1, min(most, 512)), moved=moved)
    if kind == "newmark":
        n = rng.randint(5, 24)
        return dict(kind=kind, n=n, R=log_int(8, min(256, int(2.5e6 / n ** 3))), steps=rng.randint(2, 10))
    if kind == "stress":
        n = rng.randint(5, 32)
        return dict(kind=kind, n=n, R=log_int(1, min(256, int(8.0e5 / n ** 3))), moved=rng.random() < 0.5)
    if kind == "galerkin":
        return dict(kind=kind, n=rng.randint(4, 16), m=rng.randint(2, 4), p=rng.randint(1, 3))
    return dict(kind=kind, n1=rng.randint(4, 20), n2=rng.randint(4, 20), n3=rng.randint(4, 20), n4=rng.randint(4, 20),
                n5=rng.randint(4, 20), R=log_int(4, 100))


# ------------------------------------------------------------------ inputs (plain numpy, from the seed)
def _block(nx, ny, nz, moved):
    """Model of a clamped block under unit top pressure; `moved`: interior nodes
    moved by up to 0.2 in each axis (the same mesh for every seed)."""
    model = M.clamped_block_model(nx, poisson=NU, ny=ny, nz=nz)
    if moved:
        model.xyz += _moves(nx, ny, nz)
    return model


def _moves(nx, ny, nz):
    """Displacements [nodes][3] of the interior nodes, nodes numbered x fastest."""
    rng = np.random.default_rng(100 + nx + ny + nz)
    d = np.zeros((nz + 1, ny + 1, nx + 1, 3))
    d[1:-1, 1:-1, 1:-1] = 0.2 * rng.uniform(-1, 1, (nz - 1, ny - 1, nx - 1, 3))
    return d.reshape(-1, 3)


def _germs(seed, R, terms):
    return np.random.default_rng(seed).standard_normal((R, terms))


def _moduli(seed, n):
    """Lognormal moduli of a single solve's elements (log-standard deviation 0.3)."""
    return np.exp(0.3 * np.random.default_rng(seed).standard_normal(n))


def _systems(case):
    return [(case["n1"], False), (case["n2"], False), (case["n3"], False), (case["n4"], True), (case["n5"], True)]


def _domain(case):
    return [case["nx"], case["ny"], case["nz"]]


def _sinus(case):
    return M.MassAccelerationSinusoidalLoad(1.0, 0.01, 0.01 * case["steps"], 0.1, dof=0)


def prepare(case, seed):
    ctx = M.Context(0)
    kind = case["kind"]
    s = dict(kind=kind, ctx=ctx)
    if kind == "static":
        model = _block(case["nx"], case["ny"], case["nz"], False)
        model.E_elem = _moduli(seed, model.n_elems)
        solver = M.SolverPCG(ctx, model, MAX_IT, TOL_STATIC, precision=case["precision"])
        s["model"], s["provider"] = model, M.ProblemStructural(ctx, model)
        s["static"] = M.StaticAnalyzer(s["provider"], M.LinearAnalyzer(solver))
    elif kind == "mc":
        model = _block(case["nx"], case["ny"], case["nz"], case["moved"])
        s["kl"] = M.LognormalStochasticCoefficientsProvider(_domain(case), 0.2 * case["nx"], TERMS, 16)
        s["mesh"] = M.GpuMesh(ctx, model)
        s["xi"] = torch.from_numpy(_germs(seed, case["R"], TERMS)).cuda()
        s["b"] = torch.from_numpy(model.subdomains[0].RHS).cuda()
        s["X"] = torch.empty((case["R"], model.n_dofs), dtype=torch.float64, device="cuda")
        s["tip"], s["tip_dof"] = np.zeros(case["R"]), M.tip_dof(model)
    elif kind == "newmark":
        model = _block(case["n"], case["n"], case["n"], False)
        kl = M.LognormalStochasticCoefficientsProvider([case["n"]] * 3, 0.2 * case["n"], TERMS, 12)
        an = M.NewmarkDynamicAnalyzer(ctx, model, kl, 0.25, 0.5, 0.01, 0.01 * case["steps"] + 0.001, _sinus(case),
                                      expansion_order=TERMS, simulations=case["R"], rayleigh_alpha=0.01,
                                      rayleigh_beta=0.001, max_iterations=MAX_IT, tolerance=TOL_STEP,
                                      tip_dof=model.n_dofs - 3)  # u_x of the node at the far corner
        an.RandomNumbers = _germs(seed, case["R"], TERMS)
        s["analyzer"] = an
    elif kind == "stress":
        model = _block(case["n"], case["n"], case["n"], case["moved"])
        s["mesh"] = M.GpuMesh(ctx, model)
        s["E"], s["X"] = _stress_inputs(case, seed, model.n_elems, model.n_dofs)
    elif kind == "galerkin":
        model = _block(case["n"], case["n"], case["n"], False)
        kl = M.GaussianStochasticCoefficientsProvider([case["n"]] * 3, 0.3 * case["n"], case["m"], 8, mean=2.0)
        s["op"] = M.PolynomialChaosSolverPCGMatrixCalculator(M.GpuMesh(ctx, model), kl, case["m"], case["p"])
        s["u"] = np.random.default_rng(seed).standard_normal((s["op"].PsiSize, model.n_dofs))
    elif kind == "ragged":
        batch = M.RaggedMonteCarloBatch(ctx, MAX_IT, TOL_MC)
        for i, (n, moved) in enumerate(_systems(case)):
            model = _block(n, n, n, moved)
            kl = M.LognormalStochasticCoefficientsProvider([n] * 3, 0.2 * n, TERMS, 16)
            batch.add(model, kl, _germs(seed + 1000 * i, case["R"], TERMS))
        s["batch"] = batch
    return s


def _stress_inputs(case, seed, n_elems, n_dofs):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    E = torch.exp(0.3 * torch.randn((case["R"], n_elems), dtype=torch.float64, device="cuda", generator=g))
    X = 0.01 * torch.randn((case["R"], n_dofs), dtype=torch.float64, device="cuda", generator=g)
    return E, X


def run(s):
    kind = s["kind"]
    if kind == "static":
        # one realization of the reference's loop: a new matrix for the moduli, then the solve
        s["provider"].Reset()
        s["static"].BuildMatrices()
        s["static"].Initialize()
        s["static"].Solve()
        return s["model"].subdomains[0].Solution
    if kind == "mc":
        mesh, X, tip = s["mesh"], s["X"], s["tip"]
        kl = s["kl"].struct()
        st = M.lib().MSG_MC_SOLVE_BATCH_DEVICE(
            mesh.handle, NU, ctypes.byref(kl), X.shape[0],
            s["xi"].data_ptr(), s["b"].data_ptr(), M.MSG_MODE_MIXED_BATCHED, MAX_IT, TOL_MC, s["tip_dof"], X.data_ptr(),
            tip.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None, None)
        if st != 0:
            raise RuntimeError("MSG_MC_SOLVE_BATCH_DEVICE: %d" % st)
        return {"X": X, "tip": tip}
    if kind == "newmark":
        hist = s["analyzer"].Solve()
        return {"tip": hist, "U": s["analyzer"].Solutions}
    if kind == "stress":
        eps, sig, f = M.realization_stresses(s["mesh"], s["E"], NU, s["X"])
        return {"strains": eps, "stresses": sig, "forces": f}
    if kind == "galerkin":
        return s["op"].MultiplyWithMatrix(s["u"])
    return {str(i): r["Solutions"] for i, r in enumerate(s["batch"].Solve())}


# ------------------------------------------------------------------ work
def _dofs(nx, ny, nz):
    return 3 * (nx + 1) * (ny + 1) * nz  # the z = 0 nodes are fixed


def _basis_size(m, p):
    return math.comb(m + p, p)


def work(case):
    """Inputs read once, outputs written once; the operations of one element
    product (2 x 576) for every element and realization, which no solve or
    check of one does without, and of the KL field where there is one."""
    kind = case["kind"]
    if kind == "static":
        ne, nd = case["nx"] * case["ny"] * case["nz"], _dofs(case["nx"], case["ny"], case["nz"])
        return dict(bytes=8 * (ne + 2 * nd), flops=1152 * ne)
    if kind == "mc":
        ne, nd, R = case["nx"] * case["ny"] * case["nz"], _dofs(case["nx"], case["ny"], case["nz"]), case["R"]
        return dict(bytes=8 * (R * (TERMS + nd) + nd), flops=R * ne * (1152 + 2 * TERMS))
    if kind == "newmark":
        n, R, S = case["n"], case["R"], case["steps"]
        ne, nd = n ** 3, _dofs(n, n, n)
        return dict(bytes=8 * R * (TERMS + nd + S), flops=R * ne * (1152 * S + 2 * TERMS))
    if kind == "stress":
        n, R = case["n"], case["R"]
        return dict(bytes=8 * R * (n ** 3 * (1 + 96 + 24) + _dofs(n, n, n)), flops=R * n ** 3 * 8 * (2 * 3 * 24 + 36))
    if kind == "galerkin":
        n, P = case["n"], _basis_size(case["m"], case["p"])
        return dict(bytes=16 * P * _dofs(n, n, n), flops=1152 * n ** 3 * P)
    ne, nd, R = 0, 0, case["R"]
    for n, _ in _systems(case):
        ne, nd = ne + n ** 3, nd + _dofs(n, n, n)
    return dict(bytes=8 * (R * (5 * TERMS + nd) + nd), flops=R * ne * (1152 + 2 * TERMS))


# ------------------------------------------------------------------ the same in 64 bits, without the framework
_CORNERS = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])


def _b_matrices(X):
    """X [ne][8][3] -> B [ne][8][6][24] and weights [ne][8] at the 2 x 2 x 2 Gauss points (xi outer, zeta inner)."""
    g = 1.0 / math.sqrt(3.0)
    B = np.zeros((X.shape[0], 8, 6, 24))
    w = np.zeros((X.shape[0], 8))
    for q in range(8):
        p = np.array([g if q >> 2 else -g, g if (q >> 1) & 1 else -g, g if q & 1 else -g])
        f = 1.0 + _CORNERS * p  # [8][3]
        dN = np.stack([_CORNERS[:, a] * f[:, (a + 1) % 3] * f[:, (a + 2) % 3] / 8.0 for a in range(3)])  # [3][8]
        J = np.einsum("an,enc->eac", dN, X)
        w[:, q] = np.linalg.det(J)
        d = np.einsum("eca,an->enc", np.linalg.inv(J), dN)  # dN_n/dx_c
        Bq = B[:, q].reshape(-1, 6, 8, 3)
        for c in range(3):
            Bq[:, c, :, c] = d[:, :, c]
        Bq[:, 3, :, 0], Bq[:, 3, :, 1] = d[:, :, 1], d[:, :, 0]
        Bq[:, 4, :, 1], Bq[:, 4, :, 2] = d[:, :, 2], d[:, :, 1]
        Bq[:, 5, :, 0], Bq[:, 5, :, 2] = d[:, :, 2], d[:, :, 0]
    return B, w


def _elastic():
    e1 = 1.0 / (1.0 + NU)
    e2 = e1 * NU / (1.0 - 2.0 * NU)
    D = np.full((6, 6), 0.0)
    D[:3, :3] = e2
    D[np.arange(3), np.arange(3)] = e1 + e2
    D[np.arange(3, 6), np.arange(3, 6)] = 0.5 * e1
    return D


def _stiffness(X):
    B, w = _b_matrices(X)
    return np.einsum("eq,eqrk,rs,eqsl->ekl", w, B, _elastic(), B, optimize=True)


def _cube():
    return (_CORNERS[None] + 1.0) / 2.0


class _Mesh:
    """Connectivity, free rows, load and element matrices (modulus 1) of a clamped block, on the GPU."""

    def __init__(self, nx, ny, nz, moved):
        k, j, i = (t.reshape(-1) for t in np.meshgrid(*(np.arange(n + 1) for n in (nz, ny, nx)), indexing="ij"))
        xyz = np.stack([i, j, k], axis=1).astype(np.float64)
        if moved:
            xyz += _moves(nx, ny, nz)
        base = np.arange(len(xyz)).reshape(nz + 1, ny + 1, nx + 1)
        at = (lambda c: base[c[2]:nz + c[2], c[1]:ny + c[1], c[0]:nx + c[0]].reshape(-1))
        conn = np.stack([at(c) for c in (_CORNERS + 1) // 2], axis=1)
        self.nn, self.ne = len(xyz), len(conn)
        self.X = xyz[conn]
        self.rows = torch.from_numpy((3 * conn[:, :, None] + np.arange(3)).reshape(-1)).cuda()  # [ne * 24]
        self.free = torch.from_numpy(np.flatnonzero(np.repeat(k > 0, 3))).cuda()
        lo, hi = self.X.min(axis=1), self.X.max(axis=1)
        self.centroids = lo + (hi - lo) / 2
        K = _stiffness(self.X) if moved else _stiffness(_cube())
        self.K = torch.from_numpy(K).cuda()  # [ne or 1][24][24]
        # unit pressure on the top face: a quarter of each adjacent element's face
        share = np.where((i == 0) | (i == nx), 1, 2) * np.where((j == 0) | (j == ny), 1, 2) / 4.0
        b = np.zeros((self.nn, 3))
        b[k == nz, 2] = -share[k == nz]
        self.b = torch.from_numpy(b.reshape(-1)).cuda()
        self.mask = torch.zeros(3 * self.nn, 1, dtype=torch.float64, device="cuda")
        self.mask[self.free] = 1.0

    def apply(self, E, u, K=None):
        """y [3 nn][R] = sum_e E_e K_e u_e (E [ne][R]); K: other element matrices, E None: 1."""
        K = self.K if K is None else K
        v = u[self.rows].reshape(self.ne, 24, -1)
        v = torch.matmul(K, v)
        if E is not None:
            v = v * E[:, None, :]
        return torch.zeros_like(u).index_add_(0, self.rows, v.reshape(self.ne * 24, -1))

    def diagonal(self, E, extra=None):
        d = torch.diagonal(self.K, dim1=1, dim2=2)[:, :, None] * E[:, None, :]
        if extra is not None:
            d = d + extra
        out = torch.zeros(3 * self.nn, E.shape[1], dtype=torch.float64, device="cuda")
        return out.index_add_(0, self.rows, d.reshape(self.ne * 24, -1))

    def solve(self, E, b, tol, mass=None, cK=1.0, x=None):
        """Jacobi-PCG of every column to ||r|| < tol ||b||."""
        extra = None if mass is None else torch.diagonal(mass)[None, :, None]
        E = cK * E
        A = (lambda v: self.mask * (self.apply(E, v) + (0 if mass is None else self.apply(None, v, mass))))
        dinv = 1.0 / self.diagonal(E, extra)
        b = self.mask * b
        if x is None:
            x, r = torch.zeros_like(b), b.clone()
        else:
            r = b - A(x)
        z = dinv * r
        p, rz = z.clone(), (r * z).sum(0)
        bn = b.norm(dim=0).clamp_min(1e-300)
        for it in range(20000):
            if it % 8 == 0 and float((r.norm(dim=0) / bn).max()) < tol:
                break
            q = A(p)
            a = rz / (p * q).sum(0).clamp_min(1e-300)
            x += a * p
            r -= a * q
            z = dinv * r
            new = (r * z).sum(0)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
        return x

    def out(self, x):
        return x[self.free].T.contiguous()


def _kl_terms(domain, length, terms, n1d):
    """psi's factors: the largest `terms` products of 1-D eigenpairs of exp(-|x - y| / length), by bisection."""
    c = 1.0 / length
    axes = []
    for L in domain:
        A = 0.5 * L
        pairs = []
        for k in range(1, n1d + 1):
            odd = k % 2 == 0  # sin mode
            i = k // 2
            lo, hi = ((i - 0.5) * math.pi / A, i * math.pi / A) if odd else (i * math.pi / A, (i + 0.5) * math.pi / A)
            f = ((lambda w: w * math.cos(w * A) + c * math.sin(w * A)) if odd
                 else (lambda w: c * math.cos(w * A) - w * math.sin(w * A)))
            up = f(lo + 1e-14 * (hi - lo)) > 0
            for _ in range(200):
                mid = 0.5 * (lo + hi)
                if (f(mid) > 0) == up:
                    lo = mid
                else:
                    hi = mid
            w = 0.5 * (lo + hi)
            s = math.sin(2 * w * A) / (2 * w)
            pairs.append((w, 1.0 / math.sqrt(A - s if odd else A + s), 2 * c / (w * w + c * c), odd))
        axes.append(pairs)
    top = axes[0][0][2] * axes[1][0][2] * axes[2][0][2]
    every = [(-round(axes[0][i][2] * axes[1][j][2] * axes[2][k][2] / top * 2 ** 40), i, j, k)
             for i in range(n1d) for j in range(n1d) for k in range(n1d)]
    return [(axes[0][i], axes[1][j], axes[2][k]) for _, i, j, k in sorted(every)[:terms]]


def _psi(domain, length, terms, n1d, cen):
    out = []
    for t in _kl_terms(domain, length, terms, n1d):
        f = np.full(cen.shape[0], math.sqrt(t[0][2] * t[1][2] * t[2][2]))
        for a, (w, amp, _, odd) in enumerate(t):
            x = cen[:, a] - domain[a] / 2
            f = f * amp * (np.sin(w * x) if odd else np.cos(w * x))
        out.append(f)
    return np.array(out)


def _field(domain, length, n1d, cen, xi):
    return np.exp(0.3 * xi @ _psi(domain, length, xi.shape[1], n1d, cen))  # [R][ne]


def _mc_exact(nx, ny, nz, moved, xi):
    m = _Mesh(nx, ny, nz, moved)
    E = torch.from_numpy(_field([nx, ny, nz], 0.2 * nx, 16, m.centroids, xi).T.copy()).cuda()
    parts = []
    for r in range(0, E.shape[1], 128):  # the gathered element vectors stay small
        Er = E[:, r:r + 128].contiguous()
        parts.append(m.out(m.solve(Er, m.b[:, None].expand(-1, Er.shape[1]).contiguous(), 1e-13)))
    return torch.cat(parts)


def exact(case, seed):
    kind = case["kind"]
    if kind == "static":
        m = _Mesh(case["nx"], case["ny"], case["nz"], False)
        E = torch.from_numpy(_moduli(seed, m.ne)).cuda()[:, None].contiguous()
        return m.out(m.solve(E, m.b[:, None].contiguous(), 1e-14))[0].cpu().numpy()
    if kind == "mc":
        if case["nx"] * case["ny"] * case["nz"] * case["R"] > 8.0e6:
            return None
        X = _mc_exact(case["nx"], case["ny"], case["nz"], case["moved"], _germs(seed, case["R"], TERMS))
        return {"X": X, "tip": X[:, -1].cpu().numpy()}  # u_z of the node at the far corner
    if kind == "newmark":
        return _newmark_exact(case, seed)
    if kind == "stress":
        return _stress_exact(case, seed)
    if kind == "galerkin":
        return _galerkin_exact(case, seed)
    if case["R"] * sum(n ** 3 for n, _ in _systems(case)) > 8.0e6:
        return None
    return {str(i): _mc_exact(n, n, n, moved, _germs(seed + 1000 * i, case["R"], TERMS)).cpu().numpy()
            for i, (n, moved) in enumerate(_systems(case))}


def _newmark_exact(case, seed):
    n, R, S = case["n"], case["R"], case["steps"]
    m = _Mesh(n, n, n, False)
    E = torch.from_numpy(_field([n] * 3, 0.2 * n, 12, m.centroids, _germs(seed, R, TERMS)).T.copy()).cuda()
    one = np.array([[2.0 if a == b else 1.0 for b in (-1, 1)] for a in (-1, 1)]) / 6.0
    lat = ((_CORNERS + 1) // 2).astype(int)
    Mn = np.array([[np.prod([one[lat[a][c], lat[b][c]] for c in range(3)]) for b in range(8)] for a in range(8)])
    mass = torch.from_numpy(np.kron(Mn, np.eye(3))).cuda()
    al, de, dt, ra, rb = 0.25, 0.5, 0.01, 0.01, 0.001
    a0, a1, a2 = 1 / (al * dt * dt), de / (al * dt), 1 / (al * dt)
    a3, a4, a5 = 1 / (2 * al) - 1, de / al - 1, dt * 0.5 * (de / al - 2)
    a6, a7 = dt * (1 - de), de * dt
    unit = torch.zeros(3 * m.nn, 1, dtype=torch.float64, device="cuda")
    unit[0::3] = 1.0
    fm = m.apply(None, unit, mass)
    u = torch.zeros(3 * m.nn, R, dtype=torch.float64, device="cuda")
    v, a = torch.zeros_like(u), torch.zeros_like(u)
    tip = []
    for i in range(S):
        ag = 0.1 * math.sin(2 * math.pi * dt * i)
        uu, uc = a0 * u + a2 * v + a3 * a, a1 * u + a4 * v + a5 * a
        rhs = m.mask * (m.apply(None, uu + ra * uc, mass) + rb * m.apply(E, uc) + ag * fm)
        x = m.solve(E, rhs, 2e-15, mass * (a0 + a1 * ra), 1.0 + a1 * rb, u + dt * v + (0.5 - al) * dt * dt * a)
        an = a0 * (x - u) - a2 * v - a3 * a
        v = v + a6 * a + a7 * an
        a, u = an, x
        tip.append(m.out(u)[:, len(m.free) - 3])
    return {"tip": torch.stack(tip, dim=1).cpu().numpy(), "U": m.out(u).cpu().numpy()}


def _stress_exact(case, seed):
    m = _Mesh(case["n"], case["n"], case["n"], case["moved"])
    E, X = _stress_inputs(case, seed, m.ne, len(m.free))
    B, w = (torch.from_numpy(t).cuda() for t in _b_matrices(m.X if case["moved"] else _cube()))
    B, w = B.expand(m.ne, -1, -1, -1), w.expand(m.ne, -1)
    D = torch.from_numpy(_elastic()).cuda()
    full = torch.zeros((case["R"], 3 * m.nn), dtype=torch.float64, device="cuda")
    full[:, m.free] = X
    eps, sig, f = [], [], []
    for r in range(case["R"]):
        u = full[r][m.rows].reshape(m.ne, 24)
        e = torch.einsum("eqrk,ek->eqr", B, u)
        t = torch.einsum("rs,eqs->eqr", D, e) * E[r][:, None, None]
        eps.append(e)
        sig.append(t)
        f.append(torch.einsum("eq,eqrk,eqr->ek", w, B, t))
    return {"strains": torch.stack(eps), "stresses": torch.stack(sig), "forces": torch.stack(f)}


def _multi_indices(m, p):
    """Degree by degree; within a degree in ascending lexicographic order."""
    def parts(d, k):
        if k == 1:
            return [(d,)]
        return [(i,) + t for i in range(d + 1) for t in parts(d - i, k - 1)]

    return [t for d in range(p + 1) for t in parts(d, m)]


def _galerkin_exact(case, seed):
    n, mm, p = case["n"], case["m"], case["p"]
    m = _Mesh(n, n, n, False)
    basis = _multi_indices(mm, p)
    at = {t: i for i, t in enumerate(basis)}
    P = len(basis)
    u = torch.zeros((3 * m.nn, P), dtype=torch.float64, device="cuda")
    u[m.free] = torch.from_numpy(np.random.default_rng(seed).standard_normal((P, len(m.free))).T.copy()).cuda()
    norm = [math.prod(math.factorial(q) for q in t) for t in basis]
    mean, cov = 2.0, 0.15
    psi = _psi([n] * 3, 0.3 * n, mm, 8, m.centroids)
    y = m.apply(torch.full((m.ne, 1), mean, dtype=torch.float64, device="cuda"), u) * torch.tensor(
        norm, dtype=torch.float64, device="cuda")
    for i in range(mm):
        Ku = m.apply(torch.from_numpy(mean * cov * psi[i]).cuda()[:, None], u)
        for j, t in enumerate(basis):
            for step, c in ((-1, norm[j]), (1, norm[j] * (t[i] + 1))):
                k = at.get(t[:i] + (t[i] + step,) + t[i + 1:])
                if k is not None:
                    y[:, j] += c * Ku[:, k]
    return m.out(y).cpu().numpy()
