"""The work that users of this framework have it do, as cases to time.

Every case goes through the Python binding of the C ABI (mpsdyn_b200.capi),
as the benchmark and the tests do.  The kinds:

  product   y = L W R x for a group of independent sites (the batched form of
            the effective-Hamiltonian product), operands on the device
  observe   what a program reads from a state: a local observable on every
            site and the Schmidt values of the central bond
  apply     one MPO layer applied to a state and cut back to the bond (time
            evolution by truncation)
  evolve    time steps by the variational sweep, with the observables that a
            quench records after each of them
  ground    ground states: single solves, and batches swept in lockstep in
            the mixed form that the benchmark's line uses
  excited   first excited states of a batch, above computed ground states
  serve     a stream of ground-state requests of different sizes through the
            solve server

Inputs are synthetic: seeded complex Gaussian states and environments, model
couplings of the benchmark's workloads drawn from the seed.
"""
import numpy as np
import torch

from mpsdyn_b200 import capi

SX = np.array([[0, 1], [1, 0]], dtype=complex)
SZ = np.array([[1, 0], [0, -1]], dtype=complex)
# staggered Schwinger chain: x = 1/(ag)^2 = 100, m/g = 0.125
SCHWINGER_X, SCHWINGER_MU = 100.0, 2.5


def listed():
    return [
        # one small local product: the latency of a call
        dict(name="product_one_D32", kind="product", n=1, lo=32, hi=32, w=3, mix=0),
        # the local products of one lockstep group of eight chains at the benchmark's bulk shape
        dict(name="product_group8_D128", kind="product", n=8, lo=128, hi=128, w=5, mix=0),
        # many sites of different bond dimensions in one call, odd ones among them
        dict(name="product_ragged48", kind="product", n=48, lo=32, hi=512, w=0, mix=2),
        # reading a state of the benchmark's size
        dict(name="observe_L100_D128", kind="observe", L=100, D=128),
        # one layer of an evolution by truncation
        dict(name="apply_L20_D32", kind="apply", L=20, D=32),
        # a quench while its entanglement is small: a few steps at a small bond, from the product state
        dict(name="quench_L64_D16", kind="evolve", L=64, D=16, steps=2, entangled=False),
        # one step of an entangled state at the largest bond of the quench workload
        dict(name="step_L24_D256", kind="evolve", L=24, D=256, steps=1, entangled=True),
        # the smallest whole solve: the transverse-field Ising chain of the CPU-sized configuration
        dict(name="ground_ising_L20_D20", kind="ground", model="ising", L=20, D=20, n=1, precision=0),
        # an FP64 solve of a single chain of the serving stream's middle sizes
        dict(name="ground_ising_L48_D64", kind="ground", model="ising", L=48, D=64, n=1, precision=0),
        # a lockstep group in the mixed form, at the benchmark's model and bond
        dict(name="ground_mixed8_L28_D128", kind="ground", model="schwinger", L=28, D=128, n=8, precision=1),
        # first excited states of a group, FP64
        dict(name="excited4_L20_D96", kind="excited", L=20, D=96, n=4, precision=0),
        # requests of different lengths and bonds that share the device
        dict(name="serve8_L64_D64", kind="serve", L=64, D=64, n=8, slots=4),
    ]


def _near(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["product", "product", "observe", "apply", "evolve", "ground", "ground", "excited", "serve"])
    if kind == "product":
        lo = _near(rng, 9, 128)
        return dict(kind=kind, n=_near(rng, 1, 32), lo=lo, hi=min(512, lo * rng.choice([1, 2, 4])), w=rng.choice([0, 3, 4, 5]),
                    mix=rng.randrange(1 << 20))
    if kind == "observe":
        return dict(kind=kind, L=_near(rng, 20, 100), D=_near(rng, 12, 128))
    if kind == "apply":
        return dict(kind=kind, L=rng.randrange(8, 21), D=_near(rng, 8, 32))
    if kind == "evolve":
        if rng.random() < 0.5:
            return dict(kind=kind, L=rng.randrange(20, 65), D=rng.randrange(6, 17), steps=2, entangled=False)
        return dict(kind=kind, L=rng.randrange(12, 25), D=_near(rng, 24, 256), steps=1, entangled=True)
    if kind == "ground":
        if rng.random() < 0.5:
            return dict(kind=kind, model="ising", L=rng.randrange(12, 49), D=_near(rng, 12, 64), n=1, precision=0)
        return dict(kind=kind, model="schwinger", L=2 * rng.randrange(6, 12), D=_near(rng, 24, 128), n=rng.randrange(2, 9),
                    precision=rng.choice([0, 1, 1]))
    if kind == "excited":
        return dict(kind=kind, L=2 * rng.randrange(5, 11), D=_near(rng, 16, 96), n=rng.randrange(1, 5), precision=rng.choice([0, 1]))
    return dict(kind=kind, L=rng.randrange(20, 65), D=rng.randrange(20, 65), n=rng.randrange(3, 9), slots=4)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

_context = None


def context():
    """The process's context, as a program keeps one."""
    global _context
    if _context is None:
        _context = capi.Context(0)
    return _context


class State:
    """A case's inputs and the handles that its program keeps; frees them."""

    def __init__(self, case):
        self.case, self.ctx, self.held = case, context(), []

    def hold(self, obj):
        self.held.append(obj)
        return obj

    def __del__(self):
        for obj in self.held:
            (obj.free if hasattr(obj, "free") else obj.close)()


def product_shapes(case):
    """(D, w) of every instance: fixed by the case, not by the seed."""
    rs = np.random.RandomState(case["mix"])
    shapes = []
    for _ in range(case["n"]):
        D = int(round(case["lo"] * (case["hi"] / case["lo"]) ** rs.rand()))
        if case["hi"] > case["lo"] and rs.rand() < 0.5:  # half of a mixed group: powers of two
            D = 1 << (D.bit_length() - 1)
        shapes.append((max(case["lo"], D), case["w"] or int(rs.choice([3, 5]))))
    return shapes


def product_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)

    # in memory order (slowest index first): L[a, b, a'], W[c, s, b, s'], Rt[r', c, r], x[r, s, a]
    return [dict(L=normal(D, w, D), W=normal(w, 2, w, 2), Rt=normal(D, w, D), x=normal(D, 2, D))
            for D, w in product_shapes(case)]


def gaussian_sites(L, d, D, seed):
    """Complex Gaussian site tensors A[s, a, r] of bond min(d^k, d^(L-k), D), scaled to a state of norm about 1."""
    rs = np.random.RandomState(seed & 0x7FFFFFFF)
    bond = [int(min(D, float(d) ** min(k, L - k))) for k in range(L + 1)]
    sites = []
    for a, r in zip(bond, bond[1:]):
        v = rs.standard_normal((2, d, a, r))
        sites.append((v[0] + 1j * v[1]) / np.sqrt(2.0 * d * a))
    return sites


def trotter_layer(L, J, g, dt):
    """Second-order Trotter layer exp(-i g X dt/2) exp(-i J ZZ dt) exp(-i g X dt/2) as an MPO W[u, b, s, c] of bond 2:
    exp(-i J dt z z') = cos(J dt) - i sin(J dt) z z'."""
    root = [np.sqrt(np.cos(J * dt) + 0j), np.sqrt(-1j * np.sin(J * dt))]
    half = np.cos(g * dt / 2) * np.eye(2) - 1j * np.sin(g * dt / 2) * SX
    ops = []
    for k in range(L):
        wl, wr = (1 if k == 0 else 2), (1 if k == L - 1 else 2)
        W = np.zeros((2, wl, 2, wr), dtype=complex)
        for b in range(wl):
            for c in range(wr):
                m = np.linalg.matrix_power(SZ, b + c) * (root[b] if k > 0 else 1.0) * (root[c] if k < L - 1 else 1.0)
                W[:, b, :, c] = half @ m @ half
        ops.append(W)
    return ops


def hamiltonians(s, case, rs, n):
    """n chains: Ising couplings of the paramagnet (one ground state), or Schwinger chains of different masses."""
    c = s.ctx
    if case.get("model", "schwinger") == "ising":
        return [s.hold(c.mpo_ising(case["L"], 1.0, rs.uniform(1.1, 1.5), rs.uniform(0.05, 0.2))) for _ in range(n)]
    return [s.hold(c.mpo_schwinger(case["L"], SCHWINGER_MU * rs.uniform(0.8, 1.2), SCHWINGER_X)) for _ in range(n)]


def prepare(case, seed):
    s = State(case)
    c, kind = s.ctx, case["kind"]
    rs = np.random.RandomState(seed & 0x7FFFFFFF)
    if kind == "product":
        s.inputs = product_inputs(case, seed)
        s.y = torch.zeros(sum(q["x"].numel() for q in s.inputs), dtype=torch.complex128, device="cuda")
        s.instances, at = [], 0
        for q, (D, w) in zip(s.inputs, product_shapes(case)):
            s.instances.append(dict(d=2, wl=w, wr=w, Dl=D, Dr=D, y=s.y.data_ptr() + 16 * at,
                                    **{k: v.data_ptr() for k, v in q.items()}))
            at += q["x"].numel()
        torch.cuda.synchronize()
    elif kind == "observe":
        s.psi = s.hold(c.mps(gaussian_sites(case["L"], 2, case["D"], seed)))
    elif kind == "apply":
        s.psi = s.hold(c.mps(gaussian_sites(case["L"], 2, case["D"], seed)))
        s.layer = s.hold(c.mpo(trotter_layer(case["L"], 1.0, 0.9, 0.1)))
    elif kind == "evolve":
        s.step = s.hold(c.mpo_ising_evolution(case["L"], 1.0, rs.uniform(0.2, 2.0), 0.1, 0.01, False))
        if case["entangled"]:
            s.psi = s.hold(c.mps_random_state(case["L"], 2, case["D"], seed))
        else:
            s.psi = s.hold(c.mps_product(case["L"], 2, 1))
        s.options = c.options(convtol=1e-10)
    elif kind in ("ground", "excited"):
        n = case["n"]
        s.H = hamiltonians(s, case, rs, n)
        s.starts = [s.hold(c.mps_random_state(case["L"], 2, case["D"], seed + 1000 * i)) for i in range(n)]
        s.options = c.options(convtol=1e-10, precision=case["precision"])
        if kind == "excited":
            s.levels = [s.hold(c.mps_random_state(case["L"], 2, case["D"], seed + 1000 * i + 500)) for i in range(n)]
            c.find_ground_state_batch(s.H, case["D"], s.levels, 0.0, c.options(convtol=1e-10))
    else:
        s.server = s.hold(capi.Server(0, case["slots"], 8 << 30))
        s.requests = [(capi.MODEL_ISING, int(L), int(D), 1.0, g, h, seed + i) for i, (L, D, g, h) in enumerate(
            zip(np.linspace(0.4, 1.0, case["n"]) * case["L"], np.tile([1.0, 0.5], case["n"])[:case["n"]] * case["D"],
                rs.uniform(1.1, 1.5, case["n"]), rs.uniform(0.05, 0.2, case["n"])))]
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def observables(c, psi):
    """<sigma_x> on every site and the Schmidt values of the central bond."""
    return {"sx": c.expectation_local(psi, SX), "schmidt": c.schmidt_values(psi, 0)}


def run(s):
    case, c, kind = s.case, s.ctx, s.case["kind"]
    if kind == "product":
        capi.heff_matvec_grouped(c, s.instances)
        return s.y
    if kind == "observe":
        return observables(c, s.psi)
    if kind == "apply":
        phi, discarded = s.psi.apply_mpo(s.layer, case["D"])
        out = dict(observables(c, phi), discarded=np.array([discarded]))
        phi.free()
        return out
    if kind == "evolve":
        psi, out = s.psi.copy(), []
        for _ in range(case["steps"]):
            last = psi.copy()
            c.optimize(s.step, last, psi, case["D"], s.options)
            last.free()
            out.append({"sx": c.expectation_local(psi, SX), "entropy": np.array([c.entropy(psi, case["L"] // 2)])})
        psi.free()
        return out
    if kind == "serve":
        ids = [s.server.submit(*r) for r in s.requests]
        s.server.drain()
        energy = {r["id"]: r["energy"] for r in s.server.poll()}
        return np.array([energy[i] for i in ids])
    psis = [p.copy() for p in s.starts]
    if kind == "excited":
        energies, status, _ = c.find_next_excited_state_batch(s.H, case["D"], [[lv] for lv in s.levels], psis, 0.0, s.options)
    elif case["n"] > 1:
        energies, status, _ = c.find_ground_state_batch(s.H, case["D"], psis, 0.0, s.options)
    else:
        energies, status = [c.find_ground_state(s.H[0], case["D"], psis[0], 0.0, s.options)[0]], [0]
    out = {"energy": np.array(energies), "status": np.array(status)}
    if kind == "ground" and case["precision"] == 0 and case["n"] == 1:
        out["sx"] = c.expectation_local(psis[0], SX)
    for p in psis:
        p.free()
    return out


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------

def _product_work(D, w, d=2):
    flops = 8.0 * (D * w * D * d * D + D * d * w * d * w * D + D * d * D * w * D)
    return flops, 16.0 * (2 * D * w * D + 2 * d * D * D)


def _sites(L, D, d=2):
    """(left, right) bond of every site."""
    bond = [min(D, float(d) ** min(k, L - k)) for k in range(L + 1)]
    return list(zip(bond, bond[1:]))


def _sweep_work(L, D, w, products, d=2):
    """One half-sweep: `products` local products and an environment update per site, a QR per site."""
    flops = sum((products + 1) * 8.0 * (2 * a * w * a * d * r + a * d * w * d * w * r) + 64.0 * d * a * r * r for a, r in _sites(L, D))
    return flops, sum(16.0 * (w * (a * a + r * r) + 2 * d * a * r) for a, r in _sites(L, D))


def work(case):
    """Bytes and flops of one pass.  A solve's are those of four half-sweeps with eight products a site, the least that the
    listed chains need to converge; an evolution step's those of two half-sweeps with one."""
    kind = case["kind"]
    if kind == "product":
        got = [_product_work(D, w) for D, w in product_shapes(case)]
    elif kind == "observe":
        got = [(8.0 * 6 * 2 * a * r * (a + r), 16.0 * 2 * a * r) for a, r in _sites(case["L"], case["D"])]
    elif kind == "apply":
        got = [(8.0 * 2 * (2 * r) * (2 * a) ** 2 * 4, 16.0 * 4 * a * r) for a, r in _sites(case["L"], case["D"])]
    elif kind == "evolve":
        got = [_sweep_work(case["L"], case["D"], 4, 1)] * (2 * case["steps"])
    elif kind == "serve":
        got = [_sweep_work(int(L), int(D), 3, 8) for L, D in zip(np.linspace(0.4, 1.0, case["n"]) * case["L"], np.tile([1.0, 0.5], case["n"])[:case["n"]] * case["D"])] * 4
    else:
        w = 3 if case.get("model") == "ising" else 5
        got = [_sweep_work(case["L"], case["D"], w, 8 * (2 if kind == "excited" else 1))] * (4 * case["n"])
    return {"flops": float(sum(f for f, _ in got)), "bytes": float(sum(b for _, b in got))}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch and numpy
# ---------------------------------------------------------------------------

def _left_canonical(sites):
    """QR sweep from the left; sites A[s, a, r], the last one keeps the norm."""
    out, R = [], np.eye(1)
    for A in sites:
        A = np.einsum("ab,sbr->sar", R, A)
        d, a, r = A.shape
        Q, R = np.linalg.qr(A.reshape(d * a, r))
        out.append(Q.reshape(d, a, Q.shape[1]))
    return out, R


def _observables(sites):
    left, R = _left_canonical(sites)
    norm = abs(R[0, 0])
    left[-1] = left[-1] * (R[0, 0] / norm)
    L = len(left)
    rho, sx = np.ones((1, 1)), np.zeros(L)
    pos, schmidt = L // 2, None
    tail = np.eye(1)  # right factor of the chain from the current site on
    for k in range(L - 1, -1, -1):
        A = left[k]
        sx[k] = np.einsum("sar,st,tap,rp->", A.conj(), SX, A, rho).real
        if k >= pos:  # tail' = (A tail) with its isometry taken off: the Schmidt values are those of the last factor
            d, a, r = A.shape
            B = np.einsum("sar,rq->asq", A, tail).reshape(a, -1)
            tail = np.linalg.qr(B.conj().T)[1].conj().T
            if k == pos:
                schmidt = np.sort(np.linalg.svd(tail, compute_uv=False) ** 2)
        rho = np.einsum("sar,rp,sbp->ab", A.conj(), rho, A)
    return {"sx": sx, "schmidt": schmidt}


def _apply(sites, layer, D):
    """The MPO on every site from the right, an SVD cut to D after each (the order of a right-to-left truncation)."""
    link, out, discarded = np.ones((1, 1, 1)), [], 0.0  # link[r, c, beta]
    for A, W in zip(reversed(sites), reversed(layer)):
        B = np.einsum("sar,ubsc,rcq->uabq", A, W, link, optimize=True)
        u, a, b, q = B.shape
        U, sv, Vh = np.linalg.svd(B.transpose(1, 2, 0, 3).reshape(a * b, u * q), full_matrices=False)
        keep = min(D, len(sv))
        discarded += float(np.sum(sv[keep:] ** 2))
        out.append(Vh[:keep].reshape(keep, u, q).transpose(1, 0, 2))
        link = (U[:, :keep] * sv[:keep]).reshape(a, b, keep)
    out[-1] = out[-1] * link[0, 0, 0]
    return out[::-1], discarded


def exact(case, seed):
    if case["kind"] == "product":
        # L[a, b, a'], x[r, s, a] -> T1[r, s, b, a']; W[c, s, b, s'] -> T2[r, c, s', a']; Rt[r', c, r] -> y[r', s', a']
        ys = []
        for q in product_inputs(case, seed):
            t1 = torch.einsum("abp,rsa->rsbp", q["L"], q["x"])
            t2 = torch.einsum("csbt,rsbp->rctp", q["W"], t1)
            ys.append(torch.einsum("qcr,rctp->qtp", q["Rt"], t2).reshape(-1))
        return torch.cat(ys)
    if case["kind"] == "observe":
        return _observables(gaussian_sites(case["L"], 2, case["D"], seed))
    if case["kind"] == "apply":
        phi, discarded = _apply(gaussian_sites(case["L"], 2, case["D"], seed), trotter_layer(case["L"], 1.0, 0.9, 0.1), case["D"])
        return dict(_observables(phi), discarded=np.array([discarded]))
    return None
