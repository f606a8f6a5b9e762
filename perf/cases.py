"""What is timed: the calls that a program using this engine makes, over the range of sizes it makes them at.

The engine serves an SCF program: Fock builds from integrals recomputed on the fly (direct) or from a fitted
three-index tensor (DF), in FP64 or in the split-BF16 mixed precision, for closed and open shells; nuclear gradients;
and the SCF itself.  Systems are the seeded water clusters and alkanes of ``molecular2_b200.geometry`` in the basis
sets of the library.  A case is

  kind       "direct", "uhf", "grad", "grad_df", "df", "geometry" or "scf"
  system, k  "water" (k rigid waters, randomly placed and turned) or "alkane" (C_k H_2k+2)
  basis, aux orbital basis and fitting basis (an SCF without one builds direct); spherical: pure d shells, or Cartesian ones as in older inputs
  nocc       occupied orbitals of a density (alpha ones in an open shell; beta has one less)
  storage, mixed   DF tensor layout, and the precision of the build
  side       edge of the water box in Angstrom, for one water
  host       the call on host arrays (as molecular2's Fock makes it) instead of on device pointers

``exact`` restates every result in plain torch FP64: Hermite expansions of all primitive pair densities, Coulomb
integrals between them with the Boys function from the incomplete gamma function, dense linear algebra.
"""
import math

import numpy as np
import torch

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine

PRECISION = 1e-12  # Schwarz threshold of the direct builds and gradients: the reference's default
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
AUX = {"cc-pvdz": "vdz-jkfit", "aug-cc-pvdz": "avdz-jkfit"}


def _case(kind, system, k, basis, **more):
    c = {"kind": kind, "system": system, "k": k, "basis": basis, "aux": "", "spherical": True, "nocc": 0,
         "storage": "unpacked", "mixed": False, "host": False, "side": 3.5}
    c.update(more)
    if kind in ("grad_df", "df", "geometry") or c["aux"] == "fit":
        c["aux"] = AUX[basis]
    if not c["nocc"]:
        c["nocc"] = 5 * k if system == "water" else 4 * k + 1  # electron pairs of the neutral molecule
    return c


def listed():
    return [
        # one Fock build of a single small molecule, host matrices in and out: the smallest call
        _case("direct", "water", 1, "cc-pvdz", host=True, name="direct_h2o"),
        # Fock build of a small cluster: the ordinary direct call
        _case("direct", "water", 8, "cc-pvdz", name="direct_water8"),
        # Fock build of a long chain in a triple-zeta basis: the largest direct call
        _case("direct", "alkane", 20, "6-311g**", name="direct_c20h42"),
        # open-shell Fock build, two densities, Cartesian d shells
        _case("uhf", "alkane", 6, "6-311g**", spherical=False, name="uhf_c6h14"),
        # nuclear gradient of a geometry optimisation step, four-index and density-fitted
        _case("grad", "water", 8, "cc-pvdz", host=True, name="grad_water8"),
        _case("grad_df", "water", 8, "cc-pvdz", host=True, name="grad_df_water8"),
        # DF Fock build on the resident tensor: every iteration of a DF SCF, FP64 and mixed precision
        _case("df", "water", 16, "cc-pvdz", name="df_water16"),
        _case("df", "water", 16, "cc-pvdz", mixed=True, name="df_mixed_water16"),
        # the same for systems whose tensor is kept as symmetric tiles: mixed precision streams the tiles, FP64 the
        # recomputed three-index integrals
        _case("df", "water", 24, "aug-cc-pvdz", storage="tiled", mixed=True, name="df_mixed_tiled_water24"),
        _case("df", "water", 16, "aug-cc-pvdz", storage="tiled", name="df_tiled_water16"),
        # a new geometry: engine (pairs, Schwarz bounds), fitted tensor, first build
        _case("geometry", "water", 8, "cc-pvdz", host=True, name="geometry_water8"),
        # a whole DF SCF run to tight convergence
        _case("scf", "water", 4, "cc-pvdz", aux="fit", host=True, name="scf_df_water4"),
    ]


def draw(rng):
    def size(lo, hi):
        return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo - 0.5), math.log(hi + 0.5))))))

    def case(kind, system, k, basis, **more):  # denser and looser clusters
        return _case(kind, system, k, basis, side=round(rng.uniform(3.4, 4.4), 2), **more)

    kind = rng.choice(["direct", "direct", "uhf", "grad", "grad_df", "df", "df", "tiled", "tiled", "geometry", "scf"])
    if kind in ("direct", "uhf"):
        system = rng.choice(["water", "alkane"])
        k = size(1, 14) if system == "water" else size(1, 16 if kind == "direct" else 9)
        basis = rng.choice(["cc-pvdz", "6-311g**"] if system == "alkane" or k > 6 else
                           ["cc-pvdz", "6-311g**", "aug-cc-pvdz"])
        return case(kind, system, k, basis, spherical=rng.random() < 0.7, host=rng.random() < 0.5)
    if kind == "grad":
        system = rng.choice(["water", "alkane"])
        return case(kind, system, size(1, 6 if system == "water" else 3), "cc-pvdz", spherical=rng.random() < 0.7,
                    host=True)
    if kind == "grad_df":
        return case(kind, "water", size(1, 12), "cc-pvdz", spherical=rng.random() < 0.7, host=True)
    if kind == "df":
        system = rng.choice(["water", "water", "alkane"])
        k = size(1, 20 if system == "water" else 14)
        full = 5 * k if system == "water" else 4 * k + 1
        # occupied columns: those of the molecule, or of a low-rank density change
        return case(kind, system, k, "cc-pvdz", nocc=rng.choice([full, full, rng.randint(1, full)]),
                    mixed=rng.random() < 0.5, host=rng.random() < 0.3, spherical=rng.random() < 0.8)
    if kind == "tiled":
        mixed = rng.random() < 0.5
        k = size(4, 22 if mixed else 14)
        return case("df", "water", k, "aug-cc-pvdz", storage="tiled", mixed=mixed,
                    nocc=rng.choice([5 * k, 5 * k, rng.randint(k, 5 * k)]))
    if kind == "geometry":
        return case(kind, "water", size(1, 10), rng.choice(["cc-pvdz", "aug-cc-pvdz"]), host=True)
    spherical = rng.random() < 0.7
    if rng.random() < 0.6:
        return case(kind, "water", size(1, 6), "cc-pvdz", aux="fit", host=True, spherical=spherical)
    system = rng.choice(["water", "alkane"])
    return case(kind, system, size(1, 3), rng.choice(["cc-pvdz", "6-311g**"]), host=True, spherical=spherical)


# ---------------------------------------------------------------- inputs
def _molecule(case, seed):
    if case["system"] == "alkane":
        return geometry.alkane(case["k"], seed)
    return geometry.water_cluster(case["k"], case["side"] * case["k"] ** (1 / 3), seed)


def _orbitals(basis, nocc, seed):
    """nocc orthonormal orbitals, each spread over the atoms near a centre, as the localised occupied orbitals of an
    insulator are; made on the CPU, so that every run has the same ones."""
    mol, rng = basis.mol, np.random.default_rng(seed)
    heavy = np.flatnonzero(mol.Z > 2)
    centre = heavy[np.arange(nocc) % len(heavy)]
    atom = np.repeat(basis.atom, np.diff(basis.bf_off))
    d2 = ((mol.xyz[atom][:, None, :] - mol.xyz[centre][None, :, :]) ** 2).sum(-1)
    A = torch.from_numpy(rng.normal(size=d2.shape) * np.exp(-d2 / 8.0))
    S = _overlap(basis)
    L = torch.linalg.cholesky(A.T @ (S @ A))
    return torch.linalg.solve_triangular(L, A.T, upper=False).T.contiguous().numpy()


def _inputs(case, seed):
    """(orbital basis, fitting basis or None, host arrays)"""
    mol = _molecule(case, seed)
    obs = BasisSet(mol, case["basis"], spherical=case["spherical"])
    aux = BasisSet(mol, case["aux"]) if case["aux"] else None
    h = {}
    if case["kind"] != "scf":
        C = _orbitals(obs, case["nocc"], seed)
        h["C"] = np.asfortranarray(C)
        if case["kind"] in ("direct", "grad"):
            h["D"] = np.asfortranarray(2.0 * C @ C.T)
        if case["kind"] == "uhf":  # one unpaired electron
            h["Da"], h["Db"] = (np.asfortranarray(c @ c.T) for c in (C, C[:, :-1]))
        if case["kind"] in ("grad", "grad_df"):
            h["eps"] = np.sort(-np.random.default_rng(seed + 1).uniform(0.4, 1.4, size=case["nocc"]))
            h["W"] = np.asfortranarray((C * h["eps"]) @ C.T)
    return obs, aux, h


_streams = []


def _stream():
    """The program's one stream for calls on device pointers."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0].cuda_stream


def prepare(case, seed):
    obs, aux, h = _inputs(case, seed)
    s = {"case": case, "obs": obs, "aux": aux, "h": h}
    if case["kind"] == "geometry":
        return s
    s["engine"] = eng = IntegralEngine(obs, aux)
    if aux is not None:
        eng.set_df_storage(case["storage"])
        eng.df_setup()
    if not case["host"]:
        n = eng.n
        # column-major matrices, as the C ABI takes them
        s["d"] = {k: torch.from_numpy(np.ascontiguousarray(v.T)).cuda() for k, v in h.items() if v.ndim == 2}
        s["out"] = [torch.empty(n, n, dtype=torch.float64, device=DEVICE) for _ in range(4)]
    if case["kind"] == "scf":
        s["guess"] = eng.soad_fock()
    return s


def run(state):
    case, h, eng = state["case"], state["h"], state.get("engine")
    kind, mode = case["kind"], 1 if case["mixed"] else 0
    if kind == "geometry":
        eng = IntegralEngine(state["obs"], state["aux"])
        eng.df_setup()
        J, K = eng.jk_df(h["C"])
        eng.close()
        return {"J": J, "K": K}
    if kind == "scf":
        mol = state["obs"].mol
        r, x = eng.scf_rhf(mol.nocc, mol.enuc(), df=state["aux"] is not None, maxiter=60, enconverge=1e-11, densconverge=1e-10,
                           guess_fock=state["guess"], want=True)
        return {"energy": r.energy, "D": x["D"], "eps": x["eps"]}
    if kind in ("grad", "grad_df"):
        g, g2 = (eng.compute_forces(h["D"], h["W"], PRECISION) if kind == "grad" else
                 eng.compute_forces_df(h["C"], h["eps"]))
        return {"gradient": g, "two_electron": g2}
    if case["host"]:
        if kind == "uhf":
            Ja, Jb, Ka, Kb = eng.jk_direct_uhf(h["Da"], h["Db"], PRECISION)
            return {"Ja": Ja, "Jb": Jb, "Ka": Ka, "Kb": Kb}
        J, K = eng.jk_direct(h["D"], PRECISION) if kind == "direct" else eng.jk_df(h["C"], mode)
        return {"J": J, "K": K}
    d, out, stream = state["d"], state["out"], _stream()
    if kind == "uhf":
        lib, p = eng.lib, [t.data_ptr() for t in out]
        eng._check(lib.jk_direct_uhf_device(eng.h, d["Da"].data_ptr(), d["Db"].data_ptr(), PRECISION, 1.0, *p, stream))
        return dict(zip(("Ja", "Jb", "Ka", "Kb"), out))
    if kind == "direct":
        eng.jk_direct_device(d["D"].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), PRECISION, stream=stream)
    else:
        eng.jk_df_device(d["C"].data_ptr(), case["nocc"], out[0].data_ptr(), out[1].data_ptr(), mode, stream=stream)
    return {"J": out[0], "K": out[1]}


def work(case):
    """Bytes: matrices in and out, and one read of the stored tensor.  Flops: for the contractions their own; for
    integrals a floor of 2 per Hermite integral of a significant primitive quartet and per term of the final
    transformation and digestion, the significant pairs counted with Gaussian overlaps above 1e-10."""
    mol = _molecule(case, 1)
    obs = BasisSet(mol, case["basis"], spherical=case["spherical"])
    n, o = obs.nbf, case["nocc"]
    mat = 8.0 * n * n
    herm = lambda L: (L + 1) * (L + 2) * (L + 3) / 6  # noqa: E731
    pairs = {}  # (la, lb): [primitive pairs, contracted pairs]
    types = _types(obs)
    for i, A in enumerate(types):
        for B in types[:i + 1]:
            a, b = A["exps"][:, None, :, None], B["exps"][None, :, None, :]
            d2 = ((A["xyz"][:, None] - B["xyz"][None]) ** 2).sum(-1)[:, :, None, None]
            keep = a * b / (a + b) * d2 < 23.0
            half = 0.5 if A is B else 1.0
            e = pairs.setdefault((A["l"], B["l"]), [0.0, 0.0])
            e[0] += half * float(keep.sum())
            e[1] += half * float(keep.flatten(2).any(2).sum())
    ncart = lambda l: (l + 1) * (l + 2) // 2  # noqa: E731
    direct = 0.0
    for (la, lb), (pb, cb) in pairs.items():
        for (lc, ld), (pk, ck) in pairs.items():
            comps = ncart(la) * ncart(lb) * ncart(lc) * ncart(ld)
            direct += 0.5 * (pb * pk * 2 * herm(la + lb + lc + ld) + cb * ck * comps * 14)
    if case["kind"] in ("direct", "uhf"):
        return {"bytes": 3 * mat * (2 if case["kind"] == "uhf" else 1), "flops": direct}
    if case["kind"] == "grad":
        return {"bytes": 2 * mat + 48 * mol.natom, "flops": 4 * direct}
    if not case["aux"]:  # a direct SCF of a dozen iterations
        return {"bytes": 3 * mat, "flops": 12 * (direct + 10.0 * n ** 3)}
    aux = BasisSet(mol, case["aux"])
    N = aux.nbf
    three = 0.0
    for (la, lb), (pb, cb) in pairs.items():
        for l, np_ in zip(aux.l, aux.nprim):
            three += pb * np_ * 2 * herm(la + lb + l) + cb * ncart(la) * ncart(lb) * ncart(l) * 2
    build = 2.0 * n * n * N * o + n * (n + 1.0) * N * o + 2.0 * n * n * N
    tensor = (4.0 if case["mixed"] else 8.0) * n * (n + 1) / 2 * N
    if case["kind"] == "grad_df":
        return {"bytes": 2 * mat + 48 * mol.natom, "flops": 4 * three + build}
    if case["kind"] == "df":
        if case["storage"] == "tiled" and not case["mixed"]:  # integrals recomputed, then fitted in the occupied space
            return {"bytes": 3 * mat, "flops": three + build + 1.0 * n * N * N * o}
        return {"bytes": tensor + 8.0 * n * o + 2 * mat, "flops": build}
    setup = three + N ** 3 + n * (n + 1) / 2 * N * N
    if case["kind"] == "geometry":
        return {"bytes": 8.0 * n * o + 2 * mat, "flops": setup + build}
    return {"bytes": 12 * tensor + 2 * mat, "flops": 12 * (build + 10.0 * n ** 3)}


# ---------------------------------------------------------------- plain FP64 restatement
def _dfact(k):
    return 1.0 if k <= 1 else k * _dfact(k - 2)


def _carts(l):
    return [(a, b, l - a - b) for a in range(l, -1, -1) for b in range(l - a, -1, -1)]


def _herms(L):
    return [c for k in range(L + 1) for c in _carts(k)]


def _solid(l):
    """Real solid harmonics m = -l..l over the Cartesian components, both with x^l normalised to one."""
    c, out = _carts(l), []
    r = math.sqrt
    rows = {2: [{(1, 1, 0): r(3)}, {(0, 1, 1): r(3)}, {(0, 0, 2): 1, (2, 0, 0): -0.5, (0, 2, 0): -0.5},
                {(1, 0, 1): r(3)}, {(2, 0, 0): r(3) / 2, (0, 2, 0): -r(3) / 2}],
            3: [{(2, 1, 0): 3 * r(5 / 8), (0, 3, 0): -r(5 / 8)}, {(1, 1, 1): r(15)},
                {(0, 1, 2): 4 * r(3 / 8), (2, 1, 0): -r(3 / 8), (0, 3, 0): -r(3 / 8)},
                {(0, 0, 3): 1, (2, 0, 1): -1.5, (0, 2, 1): -1.5},
                {(1, 0, 2): 4 * r(3 / 8), (3, 0, 0): -r(3 / 8), (1, 2, 0): -r(3 / 8)},
                {(2, 0, 1): r(15) / 2, (0, 2, 1): -r(15) / 2}, {(3, 0, 0): r(5 / 8), (1, 2, 0): -3 * r(5 / 8)}]}
    for row in rows[l]:
        out.append([row.get(x, 0.0) for x in c])
    return torch.tensor(out, dtype=torch.float64)


def _types(basis, device="cpu"):
    """Shells grouped by angular momentum and contraction length, coefficients normalised."""
    groups = {}
    for i in range(basis.nshell):
        groups.setdefault((int(basis.l[i]), int(basis.nprim[i]), int(basis.pure[i])), []).append(i)
    out = []
    t = lambda x: torch.as_tensor(np.asarray(x), dtype=torch.float64, device=device)  # noqa: E731
    for (l, npr, pure), idx in sorted(groups.items()):
        off = basis.prim_off[idx][:, None] + np.arange(npr)
        a, c = basis.exps[off], basis.coefs[off].copy()
        c = c * np.sqrt((4 * a) ** l * (2 * a / np.pi) ** 1.5 / _dfact(2 * l - 1))
        g = a[:, :, None] + a[:, None, :]
        s = (c[:, :, None] * c[:, None, :] * _dfact(2 * l - 1) / (2 * g) ** l * (np.pi / g) ** 1.5).sum((1, 2))
        c = c / np.sqrt(s)[:, None]
        T = _solid(l).to(device) if pure else torch.eye(len(_carts(l)), dtype=torch.float64, device=device)
        fun = torch.as_tensor(basis.bf_off[idx][:, None] + np.arange(T.shape[0]), device=device)
        out.append({"l": l, "exps": t(a), "coefs": t(c), "xyz": t(basis.mol.xyz[basis.atom[idx]]), "T": T, "fun": fun,
                    "atom": torch.as_tensor(basis.atom[idx].astype(np.int64), device=device)})
    return out


def _E(p, PA, PB, la, lb):
    """Hermite expansion of x_A^i x_B^j in one direction: [..., i, j, t]."""
    e = p.new_zeros(p.shape + (la + 1, lb + 1, la + lb + 2))
    e[..., 0, 0, 0] = 1.0
    L, h = la + lb + 1, 0.5 / p
    for i in range(la + 1):
        for j in range(lb + 1):
            if i + j == 0:
                continue
            src, X = (e[..., i - 1, 0, :], PA) if j == 0 else (e[..., i, j - 1, :], PB)
            for t in range(i + j + 1):
                v = X * src[..., t] + (t + 1) * src[..., t + 1]
                e[..., i, j, t] = v + h * src[..., t - 1] if t else v
    return e[..., :L]


def _pair_prims(A, B, la, lb):
    """Primitive pairs [sA, sB, pA, pB] of two shell types: exponents, centres, prefactor, E of x, y, z up to (la, lb)."""
    a, b = A["exps"][:, None, :, None], B["exps"][None, :, None, :]
    p = a + b
    ra, rb = A["xyz"][:, None, None, None, :], B["xyz"][None, :, None, None, :]
    P = (a[..., None] * ra + b[..., None] * rb) / p[..., None]
    K = A["coefs"][:, None, :, None] * B["coefs"][None, :, None, :] * torch.exp(-a * b / p * ((ra - rb) ** 2).sum(-1))
    E = [_E(p, P[..., x] - ra[..., x], P[..., x] - rb[..., x], la, lb) for x in range(3)]
    return a.expand(p.shape), b.expand(p.shape), p, P, K, E


def _fill(out, A, B, block, symmetric=True):
    """block [sA, sB, cart a, cart b] into out[fun, fun] as final functions."""
    v = torch.einsum("ma,nb,stab->smtn", A["T"], B["T"], block)
    out[A["fun"][:, :, None, None], B["fun"][None, None]] = v
    if symmetric:
        out[B["fun"][:, :, None, None], A["fun"][None, None]] = v.permute(2, 3, 0, 1)


def _overlap(basis):
    S = torch.zeros(basis.nbf, basis.nbf, dtype=torch.float64)
    types = _types(basis)
    for i, A in enumerate(types):
        for B in types[:i + 1]:
            a, b, p, P, K, E = _pair_prims(A, B, A["l"], B["l"])
            w = K * (math.pi / p) ** 1.5
            block = torch.empty(p.shape[:2] + (len(_carts(A["l"])), len(_carts(B["l"]))), dtype=torch.float64)
            for ia, ca in enumerate(_carts(A["l"])):
                for ib, cb in enumerate(_carts(B["l"])):
                    block[:, :, ia, ib] = (w * E[0][..., ca[0], cb[0], 0] * E[1][..., ca[1], cb[1], 0] *
                                         E[2][..., ca[2], cb[2], 0]).sum((2, 3))
            _fill(S, A, B, block)
    return S


def _shifted(E, a, la, lb, ca, cb, herms, x=None):
    """[N, na, nb, nh] products of the E of all components, or their derivative with respect to x of the first centre."""
    dev = E[0].device
    idx = lambda v, s: torch.tensor(v, device=dev).view(s)  # noqa: E731
    r = 1.0
    for d in range(3):
        i, j, t = (idx([c[d] for c in ca], (-1, 1, 1)), idx([c[d] for c in cb], (1, -1, 1)),
                   idx([h[d] for h in herms], (1, 1, -1)))
        t_in = t.clamp(max=E[d].shape[-1] - 1)
        if x == d:
            v = 2 * a[:, None, None, None] * E[d][:, i + 1, j, t_in] - i * E[d][:, (i - 1).clamp(min=0), j, t_in]
        else:
            v = E[d][:, i, j, t_in]
        r = r * (v * (t == t_in))
    return r


class _Densities:
    """Hermite expansions of the pair densities of a basis (or of its single functions), grouped by order:
    index(out, rows) says which functions a row stands for."""

    def __init__(self, obs, single=False, deriv=False, canonical=True, device=DEVICE):
        self.groups = []
        types = _types(obs, device)
        unit = {"l": 0, "exps": torch.zeros(1, 1, dtype=torch.float64, device=device),
                "coefs": torch.ones(1, 1, dtype=torch.float64, device=device), "T": torch.ones(1, 1, dtype=torch.float64, device=device)}
        for i, A in enumerate(types):
            for B in ([unit] if single else types[:i + 1] if canonical else types):
                la, lb = A["l"], B["l"]
                if single:
                    a = p = A["exps"].reshape(-1)
                    P = A["xyz"][:, None].expand(-1, A["exps"].shape[1], -1).reshape(-1, 3)
                    K = A["coefs"].reshape(-1)
                    E = [_E(p, torch.zeros_like(p), torch.zeros_like(p), la + deriv, 0)] * 3
                    seg = torch.arange(len(A["xyz"]), device=device).repeat_interleave(A["exps"].shape[1])
                    nseg = len(A["xyz"])
                else:
                    a, b, p, P, K, E = _pair_prims(A, B, la + deriv, lb)
                    seg = torch.arange(p.shape[0] * p.shape[1], device=device)
                    sa, sb = seg // p.shape[1], seg % p.shape[1]
                    nseg = len(seg)
                    seg = seg.view(p.shape[0], p.shape[1], 1, 1).expand(p.shape)
                    keep = K.abs() > 1e-20
                    if canonical and A is B:
                        keep = keep & (sa >= sb).view(p.shape[0], p.shape[1], 1, 1)
                    a, p, K, seg, P = a[keep], p[keep], K[keep], seg[keep], P[keep]
                    E = [e[keep] for e in E]
                herms = _herms(la + lb + deriv)
                M = [_shifted(E, a, la, lb, _carts(la), _carts(lb), herms, x) for x in (range(3) if deriv else [None])]
                M = torch.stack(M, 1) * K[:, None, None, None, None]  # [N, x, a, b, h]
                M = torch.einsum("ma,nb,pxabh->pxmnh", A["T"], B["T"], M).flatten(1, 3)
                fa = A["fun"] if single else A["fun"][sa]
                fb = None if single else B["fun"][sb]
                self.groups.append({"L": la + lb + deriv, "p": p, "P": P, "M": M, "seg": seg, "nseg": nseg, "fa": fa,
                                    "fb": fb, "atom": A["atom"] if single else A["atom"][sa], "nx": 3 if deriv else 1})


def _boys(L, T):
    small = T < 1e-12
    t = torch.where(small, torch.ones_like(T), T)
    a = torch.full((), L + 0.5, dtype=T.dtype, device=T.device)
    top = math.gamma(L + 0.5) * torch.special.gammainc(a, t) / (2 * t ** (L + 0.5))
    F = [torch.where(small, 1.0 / (2 * L + 1) - T / (2 * L + 3), top)]
    e = torch.exp(-T)
    for m in range(L - 1, -1, -1):
        F.append((2 * T * F[-1] + e) / (2 * m + 1))
    return F[::-1]


def _hermite_coulomb(L, alpha, d):
    """R_tuv, t + u + v <= L, of (reduced exponent, distance vectors): [..., nherm(L)]."""
    F = _boys(L, alpha * (d ** 2).sum(-1))
    R = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): (-2 * alpha) ** n * F[n]}
        for k in range(1, L - n + 1):
            for c in _carts(k):
                x = next(i for i in range(3) if c[i])
                lo = tuple(c[i] - (i == x) for i in range(3))
                v = d[..., x] * R[lo]
                if lo[x]:
                    v = v + lo[x] * R[tuple(lo[i] - (i == x) for i in range(3))]
                new[c] = v
        R = new
    return torch.stack([R[h] for h in _herms(L)], -1)


def _coulomb_blocks(X, Y, chunk=3e8):
    """(x|y) of two density groups, contracted, in row chunks of X's segments: yields (first, last, [segs, fx, segY, fy])."""
    hx, hy, L = _herms(X["L"]), _herms(Y["L"]), X["L"] + Y["L"]
    at = {h: i for i, h in enumerate(_herms(L))}
    dev = X["p"].device
    take = torch.tensor([[at[tuple(u + v for u, v in zip(a, b))] for b in hy] for a in hx], device=dev)
    sign = torch.tensor([(-1.0) ** sum(b) for b in hy], dtype=torch.float64, device=dev)
    My = Y["M"] * sign
    fx, fy = X["M"].shape[1], My.shape[1]
    nprim = torch.bincount(X["seg"], minlength=X["nseg"])
    order = torch.argsort(X["seg"], stable=True)
    ends = torch.cumsum(nprim, 0).tolist()
    cost = len(at) * 3 + len(hx) * len(hy) * 2 + fx * (len(hy) + 2 * fy)
    s0 = 0
    while s0 < X["nseg"]:
        rows, s1 = (0 if s0 == 0 else ends[s0 - 1]), s0 + 1
        while s1 < X["nseg"] and (ends[s1] - rows) * max(1, len(Y["p"])) * cost < chunk and (s1 - s0) * Y["nseg"] * fx * fy < chunk:
            s1 += 1
        x = order[rows:ends[s1 - 1]]
        out = torch.zeros(s1 - s0, Y["nseg"], fx, fy, dtype=torch.float64, device=dev)
        step = max(1, int(chunk / cost / max(1, len(x))))
        for y0 in range(0, len(Y["p"]) if len(x) else 0, step):
            y = slice(y0, y0 + step)
            p, q = X["p"][x][:, None], Y["p"][y][None]
            pref = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q))
            R = _hermite_coulomb(L, p * q / (p + q), X["P"][x][:, None] - Y["P"][y][None])
            R = (R * pref[..., None])[..., take]                       # [x, y, hx, hy]
            v = X["M"][x][:, None] @ R @ My[y][None].transpose(-1, -2)  # [x, y, fx, fy]
            part = torch.zeros(len(x), Y["nseg"], fx, fy, dtype=torch.float64, device=dev).index_add_(1, Y["seg"][y], v)
            out.index_add_(0, X["seg"][x] - s0, part)
        yield s0, s1, out
        s0 = s1


def _eri(obs):
    """(mn|rs) over all functions."""
    n, dev = obs.nbf, DEVICE
    pairs = _Densities(obs)
    I = torch.zeros(n, n, n, n, dtype=torch.float64, device=dev)
    for i, X in enumerate(pairs.groups):
        for Y in pairs.groups[:i + 1]:
            for s0, s1, v in _coulomb_blocks(X, Y):
                a, b = X["fa"][s0:s1], X["fb"][s0:s1]
                na, nb, nc, nd = a.shape[1], b.shape[1], Y["fa"].shape[1], Y["fb"].shape[1]
                v = v.view(s1 - s0, Y["nseg"], na, nb, nc, nd)
                a, b = a[:, None, :, None, None, None], b[:, None, None, :, None, None]
                c, d = Y["fa"][None, :, None, None, :, None], Y["fb"][None, :, None, None, None, :]
                used_x = (torch.bincount(X["seg"], minlength=X["nseg"])[s0:s1] > 0).view(-1, 1, 1, 1, 1, 1)
                used_y = (torch.bincount(Y["seg"], minlength=Y["nseg"]) > 0).view(1, -1, 1, 1, 1, 1)
                m = (used_x & used_y).expand(v.shape)  # segments without primitives stand for nothing
                a, b, c, d, v = a.expand(m.shape)[m], b.expand(m.shape)[m], c.expand(m.shape)[m], d.expand(m.shape)[m], v[m]
                for f in ((a, b, c, d), (b, a, c, d), (a, b, d, c), (b, a, d, c), (c, d, a, b), (d, c, a, b), (c, d, b, a), (d, c, b, a)):
                    I[f] = v
    return I


def _eri3(obs, aux):
    """(P|mn) [naux, n, n] and (P|Q)."""
    n, N, dev = obs.nbf, aux.nbf, DEVICE
    pairs, fit = _Densities(obs), _Densities(aux, single=True)
    T = torch.zeros(N, n, n, dtype=torch.float64, device=dev)
    V = torch.zeros(N, N, dtype=torch.float64, device=dev)
    for F in fit.groups:
        for X in pairs.groups:
            used = torch.bincount(X["seg"], minlength=X["nseg"]) > 0
            for s0, s1, v in _coulomb_blocks(X, F):
                u = used[s0:s1]
                a, b = X["fa"][s0:s1][u], X["fb"][s0:s1][u]
                v = v[u].view(len(a), F["nseg"], a.shape[1], b.shape[1], -1).permute(1, 4, 0, 2, 3)
                f = F["fa"][:, :, None, None, None]
                T[f, a[:, :, None], b[:, None, :]] = v
                T[f, b[:, None, :], a[:, :, None]] = v
        for G in fit.groups:
            for s0, s1, v in _coulomb_blocks(F, G):
                V[F["fa"][s0:s1][:, None, :, None], G["fa"][None, :, None, :]] = v
    return T, V


def _fitted(obs, aux):
    T, V = _eri3(obs, aux)
    n = obs.nbf
    return torch.linalg.solve_triangular(torch.linalg.cholesky(V), T.view(-1, n * n), upper=False).view(-1, n, n)


def _df_jk(B, C):
    X = B @ C                                             # [K, n, o]
    J = torch.einsum("k,kmn->mn", torch.einsum("kmo,mo->k", X, C), B)
    K = sum(x.permute(1, 0, 2).flatten(1) @ x.permute(1, 0, 2).flatten(1).T for x in X.split(256))
    return J, K


def _one_body(obs, deriv=False, device=DEVICE):
    """S, T, V; with deriv also their derivatives with respect to the first function's centre: [3, n, n] of S and T, and
    [atom, 3, n, n] of each nucleus's part of V."""
    mol, n = obs.mol, obs.nbf
    z = lambda *s: torch.zeros(*s, n, n, dtype=torch.float64, device=device)  # noqa: E731
    S, T, V, dS, dT, dV = z(), z(), z(), z(3), z(3), z(mol.natom if deriv else 0, 3)
    for A in _types(obs, device):
        for B in _types(obs, device):
            la, lb = A["l"], B["l"]
            a, b, p, P, K, E = _pair_prims(A, B, la + 1, lb + 2)
            ca, cb = _carts(la), _carts(lb)
            w = K * (math.pi / p) ** 1.5

            def overlap(d, i, j):
                return E[d][..., i, j, 0] if i >= 0 and j >= 0 else torch.zeros_like(p)

            def kinetic(d, i, j):
                return (-2 * b * b * overlap(d, i, j + 2) + b * (2 * j + 1) * overlap(d, i, j) -
                        0.5 * j * (j - 1) * overlap(d, i, j - 2))

            def block(x, kin):
                out = torch.empty(p.shape[:2] + (len(ca), len(cb)), dtype=torch.float64, device=device)
                for i, u in enumerate(ca):
                    for j, v in enumerate(cb):
                        def f(fn, d):
                            if d != x:
                                return fn(d, u[d], v[d])
                            return 2 * a * fn(d, u[d] + 1, v[d]) - u[d] * fn(d, u[d] - 1, v[d])
                        terms = [[kinetic if d == k else overlap for d in range(3)] for k in range(3)] if kin else [[overlap] * 3]
                        r = sum(f(t[0], 0) * f(t[1], 1) * f(t[2], 2) for t in terms)
                        out[:, :, i, j] = (w * r).sum((2, 3))
                return out

            for x in [None] + list(range(3 if deriv else 0)):
                _fill(S if x is None else dS[x], A, B, block(x, False), False)
                _fill(T if x is None else dT[x], A, B, block(x, True), False)
            # nuclear attraction: -Z 2 pi / p K sum E R(p, P - C)
            L, pf, Pf = la + lb + (1 if deriv else 0), p.flatten(), P.flatten(0, 3)
            M = [_shifted([e.flatten(0, 3) for e in E], a.flatten(), la, lb, ca, cb, _herms(L), x)
                 for x in [None] + list(range(3 if deriv else 0))]
            tot = 0.0
            for at in range(mol.natom):
                r = _hermite_coulomb(L, pf, Pf - torch.as_tensor(mol.xyz[at], device=device))
                r = r * (-mol.Z[at] * 2 * math.pi / pf * K.flatten())[:, None]
                v = [torch.einsum("nabh,nh->nab", m, r).view(p.shape + (len(ca), len(cb))).sum((2, 3)) for m in M]
                tot = tot + v[0]
                for x in range(3 if deriv else 0):
                    _fill(dV[at, x], A, B, v[1 + x], False)
            _fill(V, A, B, tot, False)
    return (S, T, V, dS, dT, dV) if deriv else (S, T, V)


def _by_atom(basis, per_function):
    """[3, n] per function -> [natom, 3]."""
    atom = torch.as_tensor(np.repeat(basis.atom, np.diff(basis.bf_off)).astype(np.int64), device=per_function.device)
    out = torch.zeros(basis.mol.natom, 3, dtype=torch.float64, device=per_function.device)
    return out.index_add_(0, atom, per_function.T.contiguous())


def _one_electron_gradient(obs, D, W):
    """Derivatives of tr D (T + V) - 2 tr W S and of the nuclear repulsion."""
    _, _, _, dS, dT, dV = _one_body(obs, deriv=True)
    at = torch.einsum("mn,axmn->axm", D, dV)
    g = _by_atom(obs, 2 * torch.einsum("mn,xmn->xm", D, dT) - 4 * torch.einsum("mn,xmn->xm", W, dS) + 2 * at.sum(0))
    g -= 2 * at.sum(2)  # the nuclei themselves, by translational invariance
    Z, R = torch.as_tensor(obs.mol.Z).to(DEVICE), torch.as_tensor(obs.mol.xyz).to(DEVICE)
    d = R[:, None] - R[None]
    r = d.norm(dim=-1) + torch.eye(len(Z), dtype=torch.float64, device=DEVICE)
    return g - ((Z[:, None] * Z[None] / r ** 3)[..., None] * d).sum(1)


def _direct_gradient(obs, D):
    """Two-electron part: 4 sum (1/2 D_mn D_rs - 1/4 D_mr D_ns) (m' n|rs) over all functions."""
    dpairs, pairs = _Densities(obs, deriv=True, canonical=False), _Densities(obs)
    g = torch.zeros(3, obs.nbf, dtype=torch.float64, device=DEVICE)
    for X in dpairs.groups:
        for Y in pairs.groups:
            for s0, s1, v in _coulomb_blocks(X, Y):
                m, n = X["fa"][s0:s1], X["fb"][s0:s1]
                v = v.view(s1 - s0, Y["nseg"], 3, m.shape[1], n.shape[1], Y["fa"].shape[1], Y["fb"].shape[1])
                r, t = Y["fa"], Y["fb"]
                off = 2.0 - (r[:, 0] == t[:, 0]).double()  # canonical pairs stand for both orders

                def d(x, y, dx, dy):  # D over functions x and y of [u, v, m, n, r, s], each given with its two axes
                    sx, sy = [1] * 6, [1] * 6
                    sx[dx[0]], sx[dx[1]], sy[dy[0]], sy[dy[1]] = *x.shape, *y.shape
                    return D[x.view(sx), y.view(sy)]

                M, N, R, T = (m, (0, 2)), (n, (0, 3)), (r, (1, 4)), (t, (1, 5))
                pair = lambda a, b: d(a[0], b[0], a[1], b[1])  # noqa: E731
                w = 0.5 * pair(M, N) * pair(R, T) - 0.125 * (pair(M, R) * pair(N, T) + pair(M, T) * pair(N, R))
                add = 4 * torch.einsum("uvxmnrs,uvmnrs,v->uxm", v, w, off)
                g.index_add_(1, m.flatten(), add.permute(1, 0, 2).flatten(1))
    return _by_atom(obs, g)


def _df_gradient(obs, aux, C):
    """Derivative of the DF two-electron energy 1/2 c^T V c - sum_ij (P|ij) d^P_ij, V c = (P|mn) D and V d = (P|ij)."""
    T, V = _eri3(obs, aux)
    D = 2 * C @ C.T
    inv = lambda b: torch.linalg.solve(V, b)  # noqa: E731
    Tij = torch.einsum("Pmn,mi,nj->Pij", T, C, C)
    d = inv(Tij.flatten(1)).view_as(Tij)
    c = inv(torch.einsum("Pmn,mn->P", T, D))
    W3 = c[:, None, None] * D - 2 * torch.einsum("Pij,mi,nj->Pmn", d, C, C)
    W2 = -0.5 * c[:, None] * c[None] + d.flatten(1) @ d.flatten(1).T
    g, f = (torch.zeros(3, b.nbf, dtype=torch.float64, device=DEVICE) for b in (obs, aux))
    fit, dfit = _Densities(aux, single=True), _Densities(aux, single=True, deriv=True)
    for X in _Densities(obs, deriv=True, canonical=False).groups:
        for F in fit.groups:
            for s0, s1, v in _coulomb_blocks(X, F):
                m, n = X["fa"][s0:s1], X["fb"][s0:s1]
                v = v.view(s1 - s0, F["nseg"], 3, m.shape[1], n.shape[1], -1)
                w = W3[F["fa"][None, :, None, None, :], m[:, None, :, None, None], n[:, None, None, :, None]]
                add = 2 * torch.einsum("ufxmnP,ufmnP->xum", v, w)
                g.index_add_(1, m.flatten(), add.flatten(1))
    pairs = _Densities(obs)
    for F in dfit.groups:
        for X in pairs.groups:
            for s0, s1, v in _coulomb_blocks(F, X):
                P, m, n = F["fa"][s0:s1], X["fa"], X["fb"]
                v = v.view(s1 - s0, X["nseg"], 3, P.shape[1], m.shape[1], n.shape[1])
                off = 2.0 - (m[:, 0] == n[:, 0]).double()
                w = W3[P[:, None, :, None, None], m[None, :, None, :, None], n[None, :, None, None, :]]
                f.index_add_(1, P.flatten(), torch.einsum("usxPmn,usPmn,s->xuP", v, w, off).flatten(1))
        for G in fit.groups:
            for s0, s1, v in _coulomb_blocks(F, G):
                P, Q = F["fa"][s0:s1], G["fa"]
                v = v.view(s1 - s0, G["nseg"], 3, P.shape[1], Q.shape[1])
                w = W2[P[:, None, :, None], Q[None, :, None, :]]
                f.index_add_(1, P.flatten(), 2 * torch.einsum("utxPQ,utPQ->xuP", v, w).flatten(1))
    return _by_atom(obs, g) + _by_atom(aux, f)


def _scf(obs, build, nocc, steps=60):
    """Converged closed-shell energy, density and orbital energies: DIIS from the core Hamiltonian.  build(C) gives J
    and K of C C^T."""
    S, T, V = _one_body(obs)
    H = T + V
    s, U = torch.linalg.eigh(S)
    X = U @ torch.diag(s ** -0.5) @ U.T
    R, Z = torch.as_tensor(obs.mol.xyz), torch.as_tensor(obs.mol.Z)
    enuc = sum(float(Z[i] * Z[j] / (R[i] - R[j]).norm()) for i in range(len(Z)) for j in range(i))
    F, Fs, es = H + 0.0, [], []
    for it in range(steps):
        eps, C = torch.linalg.eigh(X @ F @ X)
        C = X @ C
        J, K = build(C[:, :nocc])
        D = 2 * C[:, :nocc] @ C[:, :nocc].T
        F = H + 2 * J - K
        energy = 0.5 * float((D * (H + F)).sum()) + enuc
        e = X @ (F @ D @ S - S @ D @ F) @ X
        Fs, es = (Fs + [F])[-8:], (es + [e])[-8:]
        if float(e.abs().max()) < 1e-11:
            break
        m = len(es)
        A = torch.zeros(m + 1, m + 1, dtype=torch.float64)
        for i in range(m):
            for j in range(m):
                A[i, j] = float((es[i] * es[j]).sum())
        scale = A[m - 1, m - 1].clone()
        A[:m, :m] /= scale
        A[m, :m] = A[:m, m] = 1.0
        c = torch.linalg.lstsq(A, torch.eye(m + 1, dtype=torch.float64)[:, m:], driver="gelsd").solution[:m, 0]
        F = sum(float(x) * y for x, y in zip(c, Fs))
    return energy, D, torch.linalg.eigvalsh(X @ (H + 2 * J - K) @ X)


def exact(case, seed):
    obs, aux, h = _inputs(case, seed)
    kind, n = case["kind"], obs.nbf
    t = lambda x: torch.as_tensor(x, device=DEVICE)  # noqa: E731
    out = lambda x: x.T.cpu().numpy().T if case["host"] else x.T.contiguous()  # noqa: E731
    if kind in ("direct", "uhf"):
        if n > 200:
            return None  # minutes, and n^4 integrals beyond the memory for the largest
        I = _eri(obs)
        names = ("D",) if kind == "direct" else ("Da", "Db")
        J = [torch.einsum("mnrs,rs->mn", I, t(h[x])) for x in names]
        K = [torch.einsum("mrns,rs->mn", I, t(h[x])) for x in names]
        return dict(zip(("J", "K") if kind == "direct" else ("Ja", "Jb", "Ka", "Kb"), map(out, J + K)))
    if kind == "grad":
        if n > 100:
            return None  # minutes
        D = t(h["D"])
        g2 = _direct_gradient(obs, D)
        return {"gradient": (_one_electron_gradient(obs, D, t(h["W"])) + g2).cpu().numpy(), "two_electron": g2.cpu().numpy()}
    if kind == "grad_df":
        C = t(h["C"])
        g2 = _df_gradient(obs, aux, C)
        W = (C * t(h["eps"])) @ C.T
        return {"gradient": (_one_electron_gradient(obs, 2 * C @ C.T, W) + g2).cpu().numpy(), "two_electron": g2.cpu().numpy()}
    if kind == "scf":
        if aux is not None:
            B = _fitted(obs, aux)
            build = lambda C: _df_jk(B, C)  # noqa: E731
        elif n > 100:
            return None  # minutes
        else:
            I = _eri(obs)
            build = lambda C: [torch.einsum(x, I, C @ C.T) for x in ("mnrs,rs->mn", "mrns,rs->mn")]  # noqa: E731
        energy, D, eps = _scf(obs, build, obs.mol.nocc)
        return {"energy": energy, "D": D.cpu().numpy(), "eps": eps.cpu().numpy()}
    J, K = _df_jk(_fitted(obs, aux), t(h["C"]))
    return {"J": out(J), "K": out(K)}
