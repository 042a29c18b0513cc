"""Timed workloads of the sweep library: what a user has it do, by size.

Every case goes through the public entry points (``Engine``, ``Chain``,
``BatchEngine``).  Bond dimensions run from a few tens, where a call is a
handful of short launches, to the 1024 of the large S=1 chain; site
dimensions and MPOs are those of the spin-1/2 and spin-1 Heisenberg chains
and of the Hubbard chain.

Outputs are gauge invariant: a truncation returns the product of its two
factors (the next merge of the sweep forms such a product anyway) and the
singular values, a sweep its energies and entanglement entropy, a time step
an overlap and an expectation value.  The split-TF32 engine works to FP32
accuracy, so its results are handed on as FP32 tensors.
"""
import math

import numpy as np
import torch

from dmrgpy_gb300 import Chain, Engine
from dmrgpy_gb300 import mpo as _mpo
from dmrgpy_gb300.batch import BatchEngine

_CODE = {2: 2, 3: 3, 4: 1}      # site dimension -> site type: S=1/2, S=1, electron


def listed():
    return [
        # one Krylov step of the smallest everyday chain (bond cap 30, the
        # session default): a call is four short launches
        dict(name="matvec_chi30", kind="matvec", prec="fp64", cplx=False, chil=30, chir=30, d=2),
        # ragged mid-size FP64 matvec: bonds of a chain still growing
        dict(name="matvec_chi250_d3", kind="matvec", prec="fp64", cplx=False, chil=250, chir=203, d=3),
        # the FP64 side of the large S=1 chain
        dict(name="matvec_chi1024_d3", kind="matvec", prec="fp64", cplx=False, chil=1024, chir=1024, d=3),
        # the same bond in the split-TF32 engine
        dict(name="matvec_tf32_chi1024_d3", kind="matvec", prec="tf32x3", cplx=False, chil=1024, chir=1024, d=3),
        # environment update of the Hubbard chain, right-to-left pass
        dict(name="env_chi384_d4", kind="env", prec="fp64", cplx=False, chil=384, chir=360, d=4, side=1),
        # one bond's ground state from a random start: Krylov loop with
        # reorthogonalisation, vectors of 16k elements
        dict(name="ground_chi64", kind="ground", chi=64, d=2),
        # one two-site real-time step exp(-i tau H) in complex arithmetic
        dict(name="expm_chi96", kind="expm", chi=96, d=2),
        # FP64 truncation through the full eigenproblem
        dict(name="split_chi100", kind="split", cplx=False, chil=100, chir=100, d=2, keep=100, absorb=0),
        # FP64 truncation of a bond where the cap binds, warm start
        dict(name="subspace_chi256", kind="subspace", prec="fp64", chi=256, d=2, absorb=1),
        # whole ground-state calculation at the session's bond cap
        dict(name="gs_n16_m30", kind="gs", n=16, d=2, maxm=30, nsweeps=3),
        # many uneven Ising chains in lock step (one sweep)
        dict(name="batch_c24_n12", kind="batch", chains=24, n=12, cap=32),
        # energy and its derivative with respect to every MPO tensor
        dict(name="gradient_n24_chi64", kind="gradient", n=24, d=2, chi=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec", "tf32", "env", "env_tf32", "ground", "expm", "tdvp", "split",
                       "split_cplx", "subspace", "subspace_tf32", "gs", "batch", "gradient", "merge"])
    if kind == "matvec":
        cplx = rng.random() < 0.3
        d = rng.choice([2, 2, 3, 4])
        chi = _log(rng, 12, 320 if cplx or d == 4 else 600)
        return dict(kind="matvec", prec="fp64", cplx=cplx, chil=chi, chir=max(8, int(chi * rng.uniform(0.6, 1.0))), d=d)
    if kind == "tf32":
        d = rng.choice([2, 3, 4])
        chi = _log(rng, 64, 1000 if d < 4 else 700)
        return dict(kind="matvec", prec="tf32x3", cplx=False, chil=chi, chir=max(40, int(chi * rng.uniform(0.6, 1.0))),
                    d=d)
    if kind == "env":
        d = rng.choice([2, 3, 4])
        cplx = rng.random() < 0.3
        chi = _log(rng, 16, 256 if cplx else 480)
        return dict(kind="env", prec="fp64", cplx=cplx, chil=chi, chir=max(8, int(chi * rng.uniform(0.6, 1.0))), d=d,
                    side=rng.choice([0, 1]))
    if kind == "env_tf32":
        chi = _log(rng, 64, 1000)
        return dict(kind="env", prec="tf32x3", cplx=False, chil=chi, chir=max(40, int(chi * rng.uniform(0.6, 1.0))),
                    d=rng.choice([2, 3]), side=rng.choice([0, 1]))
    if kind == "ground":
        return dict(kind="ground", chi=_log(rng, 16, 160), d=rng.choice([2, 2, 3]))
    if kind == "expm":
        return dict(kind="expm", chi=_log(rng, 16, 128), d=2)
    if kind == "tdvp":
        return dict(kind="tdvp", n=rng.randint(8, 12), maxm=_log(rng, 10, 24), dt=rng.choice([0.02, 0.05]))
    if kind in ("split", "split_cplx"):
        cplx = kind == "split_cplx"
        d = rng.choice([2, 3])
        chi = _log(rng, 12, 64 if cplx else 110)
        chir = max(8, int(chi * rng.uniform(0.7, 1.0)))
        return dict(kind="split", cplx=cplx, chil=chi, chir=chir, d=d, keep=rng.randint(chir // 2, chi),
                    absorb=rng.choice([0, 1]))
    if kind in ("subspace", "subspace_tf32"):
        tf32 = kind == "subspace_tf32"
        return dict(kind="subspace", prec="tf32x3" if tf32 else "fp64", chi=_log(rng, 130, 800 if tf32 else 300),
                    d=rng.choice([2, 3]), absorb=rng.choice([0, 1]))
    if kind == "gs":
        return dict(kind="gs", n=rng.randint(10, 18), d=2, maxm=_log(rng, 12, 40), nsweeps=2)
    if kind == "batch":
        return dict(kind="batch", chains=rng.randint(8, 32), n=rng.randint(8, 12), cap=_log(rng, 8, 32))
    if kind == "merge":
        d = rng.choice([2, 3, 4])
        chi = _log(rng, 24, 500)
        return dict(kind="merge", chil=chi, chim=max(8, int(chi * rng.uniform(0.6, 1.0))), chir=chi, d=d)
    return dict(kind="gradient", n=rng.randint(10, 24), d=rng.choice([2, 3]), chi=_log(rng, 16, 80))


# ---------------------------------------------------------------- inputs
def _terms(n, d):
    if d < 4:
        return [(1.0 + 0j, [(op, i), (op, i + 1)]) for i in range(1, n) for op in ("Sx", "Sy", "Sz")]
    t = []
    for i in range(1, n):
        for s in ("up", "dn"):
            t.append((-1.0 + 0j, [("Cdag" + s, i), ("C" + s, i + 1)]))
            t.append((-1.0 + 0j, [("Cdag" + s, i + 1), ("C" + s, i)]))
    return t + [(4.0 + 0j, [("Nupdn", i)]) for i in range(1, n + 1)]


def _mpo_tensors(n, d):
    W, real = _mpo.build_mpo([_CODE[d]] * n, _terms(n, d))
    return W


class _Rng:
    def __init__(self, seed, cplx=False):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))
        self.dt = torch.complex128 if cplx else torch.float64

    def randn(self, *shape):
        return torch.randn(*shape, dtype=self.dt, device="cuda", generator=self.g)

    def decay(self, n, last=1e-5):
        """Schmidt-like weights from 1 down to `last`."""
        x = torch.linspace(0.0, 1.0, n, dtype=torch.float64, device="cuda") if n > 1 else torch.zeros(1, device="cuda",
                                                                                                   dtype=torch.float64)
        return torch.exp(math.log(last) * torch.sqrt(x))

    def env(self, chi, w):
        """An environment: Hermitian blocks, one channel the identity of a
        canonical state, one carrying an accumulated energy."""
        E = self.randn(chi, w, chi) / math.sqrt(chi)
        E = 0.5 * (E + E.conj().permute(2, 1, 0))
        eye = torch.eye(chi, dtype=self.dt, device="cuda")
        E[:, 0, :] = eye
        E[:, w - 1, :] = E[:, w - 1, :] - 8.0 * eye
        return E.contiguous()

    def theta(self, cl, d, cr):
        """A normalised two-site tensor with decaying Schmidt weights on both bonds."""
        t = self.randn(cl, d, d, cr)
        t = t * self.decay(cl).reshape(cl, 1, 1, 1) * self.decay(cr).reshape(1, 1, 1, cr)
        return (t / torch.linalg.vector_norm(t)).contiguous()

    def left_canonical(self, cl, d, cr):
        """(cl, d, cr) with orthonormal columns where cl d >= cr."""
        q = torch.linalg.qr(self.randn(cl * d, cr))[0] if cl * d >= cr else self.randn(cl * d, cr)
        return q.reshape(cl, d, -1).contiguous()

    def mps(self, n, d, chi):
        """Left-canonical random MPS with bond dimensions min(d^i, d^(n-i), chi)."""
        dims = [int(min(chi, d ** min(i, n - i, 40))) for i in range(n + 1)]
        out = []
        for i in range(n):
            out.append(self.left_canonical(dims[i], d, dims[i + 1]))
        return out


def _ext_left(L, W, A):
    x = torch.tensordot(L, A, dims=([2], [0]))                   # a' k s b
    x = torch.tensordot(x, W, dims=([1, 2], [0, 1]))             # a' b s' m
    x = torch.tensordot(A.conj(), x, dims=([0, 1], [0, 2]))      # b' b m
    return x.permute(0, 2, 1).contiguous()


def _ext_right(R, W, B):
    x = torch.tensordot(B, R, dims=([2], [2]))                   # a s b' m
    x = torch.tensordot(x, W, dims=([1, 3], [1, 3]))             # a b' k s'
    x = torch.tensordot(B.conj(), x, dims=([1, 2], [3, 1]))      # a' a k
    return x.permute(0, 2, 1).contiguous()


def _matvec2(L, W1, W2, R, x):
    y = torch.tensordot(L, x, dims=([2], [0]))                   # a' k s t b
    y = torch.tensordot(y, W1, dims=([1, 2], [0, 1]))            # a' t b s' m
    y = torch.tensordot(y, W2, dims=([4, 1], [0, 1]))            # a' b s' t' n
    return torch.tensordot(y, R, dims=([4, 1], [1, 2])).contiguous()


def _bond(case, seed, cplx):
    """A bond in the middle of a random chain: environments of the actual
    Hamiltonian, MPO tensors, and a random two-site tensor."""
    d, chi = case["d"], case["chi"]
    side = 1
    while d ** side < chi:
        side += 1
    n = 2 * side + 4
    r = _Rng(seed, cplx)
    W = _mpo_tensors(n, d)
    Wt = [torch.as_tensor(np.ascontiguousarray(w), device="cuda").to(r.dt) for w in W]
    half = n // 2 - 1
    one = torch.ones((1, 1, 1), dtype=r.dt, device="cuda")
    A = r.mps(n, d, chi)
    L = one
    for i in range(half):
        L = _ext_left(L, Wt[i], A[i])
    B = r.mps(n, d, chi)
    R = one
    for i in range(half):
        R = _ext_right(R, Wt[n - 1 - i], B[i].permute(2, 1, 0).contiguous())
    x = r.randn(L.shape[0], d, d, R.shape[0])
    x = (x / torch.linalg.vector_norm(x)).contiguous()
    eng = Engine(W, real=not cplx, precision="fp64")
    h = eng.heff2(L, eng.W[half], eng.W[half + 1], R, x.shape)
    return dict(eng=eng, h=h, x=x, L=L, R=R, W1=Wt[half], W2=Wt[half + 1])


def _two_site_matrix(r, m, n, last):
    """U diag(s) V^H with decaying s: (matrix, V^H, U)."""
    c = min(m, n)
    u = torch.linalg.qr(r.randn(m, c))[0]
    v = torch.linalg.qr(r.randn(n, c))[0]
    s = r.decay(c, last)
    s = s / torch.linalg.vector_norm(s)
    return ((u * s) @ v.conj().T).contiguous(), v.conj().T.contiguous(), u


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("matvec", "env"):
        d, cl, cr = case["d"], case["chil"], case["chir"]
        r = _Rng(seed, case["cplx"])
        eng = Engine(_mpo_tensors(6, d), real=not case["cplx"], precision=case["prec"])
        w = eng.W[2].shape[0]
        if kind == "matvec":
            x = r.theta(cl, d, cr)
            L, R = r.env(cl, w), r.env(cr, w)
            return dict(case=case, eng=eng, x=x, h=eng.heff2(L, eng.W[2], eng.W[3], R, x.shape), L=L, R=R)
        if case["side"] == 0:
            A = r.left_canonical(cl, d, cr)
            E = r.env(cl, w)
        else:
            A = r.left_canonical(cr, d, cl).permute(2, 1, 0).contiguous()
            E = r.env(cr, w)
        return dict(case=case, eng=eng, A=A, E=E)
    if kind in ("ground", "expm"):
        return dict(case=case, **_bond(case, seed, kind == "expm"))
    if kind == "merge":
        r = _Rng(seed)
        eng = Engine(_mpo_tensors(4, case["d"]), real=True, precision="fp64")
        A = r.left_canonical(case["chil"], case["d"], case["chim"])
        B = r.randn(case["chim"], case["d"], case["chir"]) * r.decay(case["chim"]).reshape(-1, 1, 1)
        return dict(case=case, eng=eng, A=A, B=B.contiguous())
    if kind == "split":
        r = _Rng(seed, case["cplx"])
        eng = Engine(_mpo_tensors(4, case["d"]), real=not case["cplx"], precision="fp64")
        M = _two_site_matrix(r, case["chil"] * case["d"], case["d"] * case["chir"], 1e-4)[0]
        return dict(case=case, eng=eng, M=M)
    if kind == "subspace":
        r = _Rng(seed)
        eng = Engine(_mpo_tensors(4, case["d"]), real=True, precision=case["prec"])
        k = case["chi"]
        m = k * case["d"]
        M, Vh, U = _two_site_matrix(r, m, m, 1e-4)
        # the neighbour tensor of the last pass: close to, not equal to, the
        # leading singular vectors
        near = (Vh[:k].T if case["absorb"] == 0 else U[:, :k]) + 1e-3 * r.randn(m, k) / math.sqrt(m)
        q = torch.linalg.qr(near)[0]
        start = q.T.contiguous() if case["absorb"] == 0 else q.contiguous()
        return dict(case=case, eng=eng, M=M, start=start)
    if kind == "gs":
        c = Chain([_CODE[case["d"]]] * case["n"])
        c.set_sweep_params(case["maxm"], case["nsweeps"], 1e-12, 0.0)
        c.set_hamiltonian(_terms(case["n"], case["d"]))
        np.random.seed(seed % (1 << 31))
        return dict(case=case, chain=c, wf=c.random_mps())
    if kind == "tdvp":
        n = case["n"]
        c = Chain([2] * n)
        c.set_sweep_params(case["maxm"], 1, 1e-10, 0.0)
        np.random.seed(seed % (1 << 31))
        H = c.build_operator(_terms(n, 2))
        # a product state of random directions: bonds grow during the step
        sp = np.random.randn(n, 2) + 1j * np.random.randn(n, 2)
        sp /= np.linalg.norm(sp, axis=1, keepdims=True)
        from dmrgpy_gb300 import MPS
        wf = MPS([sp[i].reshape(1, 2, 1) for i in range(n)], center=1)
        for _ in range(2):
            wf = c.tdvp_step(H, wf, case["dt"])
        return dict(case=case, chain=c, H=H, wf=wf)
    if kind == "batch":
        rng = np.random.default_rng(seed)
        n, C = case["n"], case["chains"]
        hs = rng.uniform(0.5, 1.5, C)
        caps = [max(4, case["cap"] >> int(k)) for k in rng.integers(0, 3, C)]
        Ws = [_mpo.build_mpo([2] * n, [(-1.0 + 0j, [("Sz", i), ("Sz", i + 1)]) for i in range(1, n)]
                             + [(complex(h), [("Sx", i)]) for i in range(1, n + 1)])[0] for h in hs]
        be = BatchEngine(Ws, real=True)
        As = be.random_states([2] * n, 4, seeds=[int(s) for s in rng.integers(0, 1 << 30, C)])
        be.canonicalize(As)
        return dict(case=case, be=be, As=As, caps=caps)
    if kind == "gradient":
        r = _Rng(seed)
        eng = Engine(_mpo_tensors(case["n"], case["d"]), real=True, precision="fp64")
        return dict(case=case, eng=eng, A=r.mps(case["n"], case["d"], case["chi"]))
    raise ValueError(kind)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "matvec":
        y = state["eng"].apply(state["h"], state["x"])
        return y if case["prec"] == "fp64" else y.to(torch.float32)
    if kind == "env":
        eng = state["eng"]
        f = eng.env_left if case["side"] == 0 else eng.env_right
        y = f(state["E"], eng.W[2], state["A"])
        return y if case["prec"] == "fp64" else y.to(torch.float32)
    if kind == "ground":
        x = state["x"].clone()
        e, _ = state["eng"].ground(state["h"], x, 2)
        return [np.array([e]), x]
    if kind == "expm":
        x = state["x"].clone()
        state["eng"].expm(state["h"], x, -0.025j, 50)
        return x
    if kind == "merge":
        return state["eng"].merge(state["A"], state["B"])
    if kind == "split":
        eng, M = state["eng"], state["M"]
        lo, ro, s, keep, _ = eng.svd(M, 0.0, case["keep"], 1, case["absorb"])
        return [eng.gemm(lo, ro), s[:keep], keep]
    if kind == "subspace":
        eng, M = state["eng"], state["M"]
        lo, ro, _, keep, _ = eng.subspace_split(M, case["chi"], state["start"], case["chi"], case["absorb"], 0.0)
        y = eng.gemm(lo, ro)
        return [y if case["prec"] == "fp64" else y.to(torch.float32), keep]
    if kind == "gs":
        c = state["chain"]
        c.set_wavefunction(state["wf"])
        e = c.gs_energy()
        return np.array([e, c.bond_entropy(c.gs_wavefunction(), case["n"] // 2)])
    if kind == "tdvp":
        c, wf = state["chain"], state["wf"]
        out = c.tdvp_step(state["H"], wf, case["dt"])
        return np.array([c.overlap(wf, out), c.vev([(1.0 + 0j, [("Sz", case["n"] // 2)])], out)])
    if kind == "batch":
        e, _ = state["be"].sweep([list(A) for A in state["As"]], state["caps"], 0.0)
        return np.asarray(e)
    if kind == "gradient":
        e, G = state["eng"].mpo_gradients(state["A"])
        return [np.array([e])] + list(G)
    raise ValueError(kind)


# ---------------------------------------------------------------- the unavoidable work of a pass
def _w(d):
    return {2: 5, 3: 5, 4: 6}[d]


def _split_work(m, n, k, es, real):
    c = min(m, n)
    return dict(bytes=es * (2 * m * n + k * (m + n)), flops=(4.0 * m * n * c + 2.0 * m * n * k) * (1 if real else 4))


def work(case):
    kind = case["kind"]
    if kind == "matvec":
        cl, cr, d = case["chil"], case["chir"], case["d"]
        w = _w(d)
        es = 16 if case["cplx"] else 8
        return dict(bytes=es * (w * (cl * cl + cr * cr) + 2 * cl * d * d * cr),
                    flops=Engine.heff2_flops(cl, d, d, cr, w, w, w, case["cplx"]))
    if kind == "env":
        cl, cr, d = case["chil"], case["chir"], case["d"]
        w = _w(d)
        es = 16 if case["cplx"] else 8
        macs = cl * cr * d * w * (cl + cr) + cl * cr * d * d * w * w
        return dict(bytes=es * (w * (cl * cl + cr * cr) + cl * d * cr), flops=2.0 * macs * (4 if case["cplx"] else 1))
    if kind in ("ground", "expm"):
        chi, d = case["chi"], case["d"]
        w = _w(d)
        its = 40 if kind == "ground" else 8       # Krylov steps such a start takes
        f = its * Engine.heff2_flops(chi, d, d, chi, w, w, w, kind == "expm")
        es = 16 if kind == "expm" else 8
        return dict(bytes=es * (2 * w * chi * chi + 2 * chi * chi * d * d), flops=f)
    if kind == "merge":
        a, b, c, d = case["chil"], case["chim"], case["chir"], case["d"]
        return dict(bytes=8.0 * (a * d * b + b * d * c + a * d * d * c), flops=2.0 * a * d * b * d * c)
    if kind == "split":
        return _split_work(case["chil"] * case["d"], case["d"] * case["chir"], case["keep"], 16 if case["cplx"] else 8,
                           not case["cplx"])
    if kind == "subspace":
        m, k = case["chi"] * case["d"], case["chi"]
        return dict(bytes=8.0 * (2 * m * m + 3 * m * k), flops=6.0 * m * m * k + 4.0 * m * k * k)
    if kind == "gs":
        chi, n, d = case["maxm"], case["n"], case["d"]
        bonds = 2 * (n - 1) * case["nsweeps"]
        per = 4 * Engine.heff2_flops(chi, d, d, chi, 5, 5, 5) + 4.0 * (chi * d) ** 3
        return dict(bytes=16.0 * n * chi * chi * d, flops=bonds * per)
    if kind == "tdvp":
        chi, n, d = case["maxm"], case["n"], 2
        per = 6 * Engine.heff2_flops(chi, d, d, chi, 5, 5, 5, True) + 16.0 * (chi * d) ** 3
        return dict(bytes=32.0 * n * chi * chi * d, flops=2 * (n - 1) * per)
    if kind == "batch":
        chi, n, d = case["cap"] / 2, case["n"], 2
        per = 6 * Engine.heff2_flops(chi, d, d, chi, 3, 3, 3) + 4.0 * (chi * d) ** 3
        return dict(bytes=16.0 * n * chi * chi * d * case["chains"], flops=case["chains"] * 2 * (n - 1) * per)
    chi, n, d = case["chi"], case["n"], case["d"]
    w = _w(d)
    one = 2.0 * (2 * chi ** 3 * d * w + chi * chi * d * d * w * w)
    return dict(bytes=8.0 * n * (chi * chi * d + d * d * w * w), flops=3 * n * one)


# ---------------------------------------------------------------- the values, in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind in ("gs", "tdvp", "batch"):
        return None                     # a whole variational sweep: no value but its own
    s = prepare(case, seed)
    if kind == "matvec":
        eng = s["eng"]
        return _matvec2(s["L"], eng.W[2], eng.W[3], s["R"], s["x"])
    if kind == "env":
        f = _ext_left if case["side"] == 0 else _ext_right
        return f(s["E"], s["eng"].W[2], s["A"])
    if kind == "merge":
        return torch.tensordot(s["A"], s["B"], dims=([2], [0]))
    if kind == "ground":
        return [np.array([_lowest(s)]), None]
    if kind == "expm":
        y, term = s["x"].clone(), s["x"]
        for k in range(1, 60):
            term = _matvec2(s["L"], s["W1"], s["W2"], s["R"], term) * (-0.025j / k)
            y = y + term
            if float(torch.linalg.vector_norm(term)) < 1e-18:
                break
        return y
    if kind == "split":
        u, sv, vh = torch.linalg.svd(s["M"], full_matrices=False)
        k = min(case["keep"], sv.numel())
        return [(u[:, :k] * sv[:k]) @ vh[:k], sv[:k], None]
    if kind == "subspace":
        M = s["M"]
        if case["absorb"] == 0:
            q = torch.linalg.qr(M @ s["start"].T)[0]
            return [q @ (q.T @ M), None]
        q = torch.linalg.qr(M.T @ s["start"])[0]
        return [(M @ q) @ q.T, None]
    eng, A = s["eng"], s["A"]
    n = len(A)
    one = torch.ones((1, 1, 1), dtype=torch.float64, device="cuda")
    R = {n: one}
    for i in range(n - 1, 0, -1):
        R[i] = _ext_right(R[i + 1], eng.W[i], A[i])
    L, nrm, G = one, torch.ones((1, 1), dtype=torch.float64, device="cuda"), []
    for i in range(n):
        x = torch.tensordot(L, A[i], dims=([2], [0]))                       # a' k s b
        x = torch.tensordot(x, R[i + 1], dims=([3], [2]))                   # a' k s b' m
        G.append(torch.tensordot(x, A[i], dims=([0, 3], [0, 2])).permute(0, 1, 3, 2))   # k s m s' -> k s s' m
        L = _ext_left(L, eng.W[i], A[i])
        nrm = torch.tensordot(A[i], torch.tensordot(nrm, A[i], dims=([1], [0])), dims=([0, 1], [0, 1]))
    nn = float(nrm.reshape(-1)[0])
    return [np.array([float(L.reshape(-1)[0]) / nn])] + [g.contiguous() / nn for g in G]


def _lowest(s):
    """Lowest eigenvalue by Lanczos with full reorthogonalisation, run past convergence."""
    x = s["x"].reshape(-1)
    q = x / torch.linalg.vector_norm(x)
    Q = q.reshape(1, -1)
    al, be, last = [], [], None
    for it in range(min(300, x.numel())):
        w = _matvec2(s["L"], s["W1"], s["W2"], s["R"], Q[-1].reshape(s["x"].shape)).reshape(-1)
        al.append(float(torch.dot(Q[-1], w)))
        for _ in range(2):
            w = w - Q.T @ (Q @ w)
        b = float(torch.linalg.vector_norm(w))
        e = float(np.linalg.eigvalsh(np.diag(al) + np.diag(be, 1) + np.diag(be, -1))[0])
        if b < 1e-12 or (last is not None and abs(e - last) < 1e-15 * abs(e)):
            return e
        last = e
        be.append(b)
        Q = torch.cat([Q, (w / b).reshape(1, -1)])
    return last
