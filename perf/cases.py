"""Performance cases: what a program that uses this framework has it compute.

Every case goes through the package's public entry points on seeded synthetic
systems (rigid waters on a lattice or in a box at 1.0 g/cm^3, staggered linear
alkanes).  A case is a dict with a "kind" and a size:

  single_point   a molecule, alone, solvated or a cluster, from its coordinates
                 to its heat and density: context, integrals, SCF with the
                 default keywords, density back on the host.  The call of a
                 geometry scan or a conformer search, one small molecule at a
                 time: latency.
  scf            the SCF of a context that keeps its integrals on the device
                 (iter), in one of the modes it is run in:
                   plain  default keywords: FP64, a full diagonalisation in
                          every iteration;
                   pulay  FP64, pseudo-diagonalisation and Pulay's converger;
                   fast   learned starting density, SHIFT=0, pseudo-
                          diagonalisation, Pulay, split-precision tensor-core
                          products and the FP64 finish.
  batch          heats of many small molecules in one launch (screening).
  mozyme         the localized-orbital SCF from its starting LMOs.
  fock           one two-electron Fock build (fock2), called on device arrays.
  diagonalise    a Fock matrix to its eigenvalues and closed-shell density, the
                 two steps iter takes in every plain iteration.
  pseudo_step    one pseudo-diagonalisation (Fmo product and the ordered 2x2
                 rotation sweep) and the density of the rotated vectors, the
                 steps of a pseudo-diagonalising iteration.
  gradient       dcart's Cartesian gradient at a given density.
  train          training steps of the starting-density networks (forward,
                 backward, Adam), then the parameters read back.

listed() holds one or two sizes of each kind, draw(rng) gives another of the
same ranges.  Orders are not multiples of a tile: 6 per water, 6k + 2 for an
alkane, any number for a diagonalisation.
"""
import math

import numpy as np
import torch

from mopac_gpu_b200 import guess as guess_mod
from mopac_gpu_b200 import kernels, mozyme, workloads
from mopac_gpu_b200._lib import lib
from mopac_gpu_b200.batch import Batch
from mopac_gpu_b200.scf import ScfContext

# kind -> size range of draw()
RANGES = {
    "alkane": (3, 20),          # carbons: the batched workload's molecules
    "solvent": (1, 60),         # waters around it, or alone
    "plain": (48, 120),
    "pulay": (48, 240),
    "fast": (64, 400),
    "batch": (32, 2000),        # molecules
    "mozyme": (48, 220),
    "fock": (24, 512),
    "diagonalise": (48, 3072),  # matrix order
    "pseudo_step": (48, 500),
    "gradient": (24, 256),
    "train": (512, 4096),       # rows of a minibatch
}


def listed():
    return [
        # hexane alone, 38 orbitals: the smallest call, all latency
        {"name": "single_point_hexane", "kind": "single_point", "carbons": 6, "waters": 0},
        # a 24-water cluster, 144 orbitals: an ordinary single molecule
        {"name": "single_point_water24", "kind": "single_point", "carbons": 0, "waters": 24},
        # default keywords on a 600-orbital cluster: a full eigensolve per iteration
        {"name": "scf_plain_water100", "kind": "scf", "mode": "plain", "size": 100},
        # FP64 convergers on a 1026-orbital cluster
        {"name": "scf_pulay_water171", "kind": "scf", "mode": "pulay", "size": 171},
        # the benchmark's flagship step: the 3072-orbital water box, fast mode
        {"name": "scf_fast_box512", "kind": "scf", "mode": "fast", "size": 512},
        # screening: 1500 alkanes C3..C20 in one call
        {"name": "batch_alkanes1500", "kind": "batch", "size": 1500},
        # localized-orbital SCF of a 150-water box
        {"name": "mozyme_water150", "kind": "mozyme", "size": 150},
        # one Fock build, 1998 orbitals
        {"name": "fock_water333", "kind": "fock", "size": 333},
        # odd matrix order
        {"name": "diagonalise_1501", "kind": "diagonalise", "size": 1501},
        # one pseudo-diagonalisation step at 2046 orbitals
        {"name": "pseudo_step_water341", "kind": "pseudo_step", "size": 341},
        # forces of a 600-atom cluster
        {"name": "gradient_water200", "kind": "gradient", "size": 200},
        # training: four steps of 2048 rows for each of the five networks
        {"name": "train_2048", "kind": "train", "size": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single_point", "single_point", "scf", "scf", "scf", "batch", "mozyme", "fock",
                       "diagonalise", "pseudo_step", "gradient", "train"])
    if kind == "single_point":
        carbons, waters = _log_int(rng, *RANGES["alkane"]), _log_int(rng, *RANGES["solvent"])
        alone = rng.choice(["alkane", "waters", "solvated", "solvated"])
        return {"kind": kind, "carbons": 0 if alone == "waters" else carbons,
                "waters": 0 if alone == "alkane" else waters}
    if kind == "scf":
        mode = rng.choice(["plain", "pulay", "fast"])
        return {"kind": kind, "mode": mode, "size": _log_int(rng, *RANGES[mode])}
    return {"kind": kind, "size": _log_int(rng, *RANGES[kind])}


# ------------------------------------------------------------------ inputs
class _ContextArray:
    """A context's device array as torch takes it: the tensor keeps this object,
    and with it the context that owns the memory."""

    def __init__(self, ctx, name, count):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "version": 3, "strides": None,
                                         "data": (ctx.device_ptrs()[name], False)}


def _view(ctx, name, count):
    return torch.as_tensor(_ContextArray(ctx, name, count), device="cuda")


def _orbitals(nat):
    return np.where(np.asarray(nat) == 1, 1, 4)


def _alkanes(count, rng, distinct=96):
    """`count` alkanes C3..C20: `distinct` conformers, the others the same
    conformers with every atom displaced by up to 0.02 A per axis."""
    lo, hi = RANGES["alkane"]
    base = [workloads.alkane(int(rng.integers(lo, hi + 1)), rng) for _ in range(min(count, distinct))]
    out = list(base)
    while len(out) < count:
        nat, xyz = base[int(rng.integers(len(base)))]
        out.append((nat, xyz + rng.uniform(-0.02, 0.02, size=xyz.shape)))
    return out


def _molecule(carbons, waters, rng):
    """An alkane conformer with its atoms displaced by up to 0.02 A per axis,
    and rigid waters on the lattice points around it, nearest first."""
    nat, xyz = np.zeros(0, np.int32), np.zeros((0, 3))
    if carbons:
        nat, xyz = workloads.alkane(carbons, rng)
        xyz = xyz - xyz.mean(axis=0) + rng.uniform(-0.02, 0.02, size=xyz.shape)
    if waters:
        edge = 3.1 * np.arange(-8, 9)
        site = np.stack(np.meshgrid(edge, edge, edge, indexing="ij"), axis=-1).reshape(-1, 3)
        site = site + rng.uniform(-0.15, 0.15, size=site.shape)
        near = np.full(len(site), np.inf) if not carbons else \
            np.linalg.norm(site[:, None] - xyz[None], axis=-1).min(axis=1)
        order = np.argsort(near if carbons else np.linalg.norm(site, axis=1), kind="stable")
        site = site[order][near[order] > 3.2][:waters]
        shape, one = workloads.water_lattice(1, seed=int(rng.integers(1 << 30)), jitter=0.0)
        turn = np.linalg.qr(rng.normal(size=(waters, 3, 3)))[0]
        turn = turn * np.sign(np.linalg.det(turn))[:, None, None]
        water = site[:, None] + np.einsum("wij,aj->wai", turn, one - one[0])
        nat = np.concatenate([nat, np.tile(shape, waters)]).astype(np.int32)
        xyz = np.concatenate([xyz, water.reshape(-1, 3)])
    return nat, xyz


def _density(nat, xyz, gen):
    """A packed density of the shape an SCF meets: the atoms' valence
    populations on the diagonal, plus symmetric elements that fall off with
    the distance of their atoms."""
    nor = _orbitals(nat)
    atom = torch.from_numpy(np.repeat(np.arange(len(nat)), nor)).cuda()
    pop = np.repeat(np.where(np.asarray(nat) == 1, 1.0, np.where(np.asarray(nat) == 6, 4.0, 6.0) / 4.0), nor)
    n = int(nor.sum())
    r = torch.from_numpy(np.asarray(xyz, np.float64).reshape(-1, 3)).cuda()
    fall = torch.exp(-torch.cdist(r, r, compute_mode="donot_use_mm_for_euclid_dist") / 1.2)
    noise = torch.randn((n, n), generator=gen, dtype=torch.float64, device="cuda")
    p = 0.05 * noise * fall[atom][:, atom]
    p = p + p.T + torch.diag(torch.from_numpy(pop).cuda())
    i, j = torch.tril_indices(n, n, device="cuda")
    return p[i, j].contiguous()


def _fock_inputs(waters, seed):
    """(context, atoms, h, w, ptot, pa) of a water lattice on the device."""
    nat, xyz = workloads.water_lattice(waters, seed=seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    ctx = ScfContext(nat, xyz)
    ctx.hcore()
    nor = _orbitals(nat)
    last = np.cumsum(nor)
    atoms = kernels.Atoms(last - nor + 1, last)
    p = _density(nat, xyz, gen)
    return ctx, atoms, _view(ctx, "h", ctx.mpack), _view(ctx, "w", ctx.n2elec), p, p * 0.5


def _fock_matrix(order, seed):
    """The leading `order` rows of a water lattice's Fock matrix, packed."""
    ctx, atoms, h, w, p, pa = _fock_inputs(-(-order // 6), seed)
    f = torch.empty_like(p)
    kernels.fock2(atoms, f, h, p, pa, w)
    return f[:order * (order + 1) // 2].clone()


def _full(packed, n):
    a = torch.zeros((n, n), dtype=torch.float64, device=packed.device)
    i, j = torch.tril_indices(n, n, device=packed.device)
    a[i, j] = packed
    a[j, i] = packed
    return a


def prepare(case, seed):
    kind, size = case["kind"], case.get("size")
    rng = np.random.default_rng(seed)
    if kind == "single_point":
        nat, xyz = _molecule(case["carbons"], case["waters"], rng)
        return {"kind": kind, "nat": nat, "xyz": xyz}
    if kind == "scf":
        mode = case["mode"]
        state = {"kind": kind, "mode": mode}
        if mode == "fast":
            nat, xyz, _ = workloads.water_box(size, seed=seed)
            state["model"] = guess_mod.GuessModel(path=guess_mod.BOX_MODEL)
        else:
            nat, xyz = workloads.water_lattice(size, seed=seed)
        ctx = ScfContext(nat, xyz)
        ctx.hcore()
        state.update(ctx=ctx, p=_view(ctx, "p", ctx.mpack), eigs=_view(ctx, "eigs", ctx.norbs))
        return state
    if kind == "batch":
        return {"kind": kind, "batch": Batch(_alkanes(size, rng))}
    if kind == "mozyme":
        # one box per size, turned and its molecules reordered by the seed: the
        # stored pairs are then as many for every seed
        nat, xyz, _ = workloads.water_box(size)
        turn = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        xyz = (xyz.reshape(-1, 3, 3)[rng.permutation(size)] @ (turn * np.sign(np.linalg.det(turn))).T).reshape(-1, 3)
        layout = mozyme.Layout(_orbitals(nat).astype(np.int32), xyz, 81.0, 8.9 ** 2)  # CUTOFF=9
        coord = torch.from_numpy(np.ascontiguousarray(xyz, np.float64)).cuda()
        h, w, enuclr = mozyme.hcore(layout, torch.from_numpy(np.ascontiguousarray(nat, np.int32)).cuda(), coord)
        _, occ, vir = mozyme.water_lmos(nat, xyz, pad_atoms=400)
        nat = np.ascontiguousarray(nat, np.int32)
        return {"kind": kind, "layout": layout, "coord": coord, "h": h, "w": w, "enuclr": enuclr, "occ": occ,
                "vir": vir, "atheat": lib().mb_atheat(nat.size, nat.ctypes.data)}
    if kind == "fock":
        ctx, atoms, h, w, p, pa = _fock_inputs(size, seed)
        return {"kind": kind, "ctx": ctx, "atoms": atoms, "h": h, "w": w, "p": p, "pa": pa, "f": torch.empty_like(p)}
    if kind == "diagonalise":
        return {"kind": kind, "f": _fock_matrix(size, seed), "nocc": 2 * size // 3}
    if kind == "pseudo_step":
        n = 6 * size
        f = _fock_matrix(n, seed)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed + 1)
        eigs, c = torch.linalg.eigh(_full(f, n))
        # the next iteration's matrix: a density step later, elements moved by up to about 1e-2 eV
        step = 1.0e-3 * torch.randn(f.shape, generator=gen, dtype=torch.float64, device="cuda")
        return {"kind": kind, "f": f + step, "c": c.T.contiguous(), "eigs": eigs, "nocc": 4 * size}
    if kind == "gradient":
        nat, xyz = workloads.water_lattice(size, seed=seed)
        ctx = ScfContext(nat, xyz)
        ctx.hcore()
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        _view(ctx, "p", ctx.mpack).copy_(_density(nat, xyz, gen))
        return {"kind": kind, "ctx": ctx}
    if kind == "train":
        nat, xyz = workloads.water_lattice(125, seed=seed)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        pairs = guess_mod.PairSet(nat, xyz)
        targets = pairs.targets(_density(nat, xyz, gen).data_ptr())
        trainer = guess_mod.Trainer(guess_mod.init_blob(seed), size)
        sets = []
        for t in range(guess_mod.NTYPES):
            a, b = pairs.offsets[t], pairs.offsets[t + 1]
            raw, y = pairs.feat[a:b], targets[a:b]
            std = raw.std(0).cpu().numpy()
            trainer.set_norm(t, raw.mean(0).cpu().numpy(), np.where(std > 1.0e-3, std, 1.0),
                             np.zeros(guess_mod.DOUT), np.ones(guess_mod.DOUT))
            pick = torch.randint(b - a, (4 * size,), generator=gen, device="cuda")
            raw = raw[pick] * (1.0 + 0.01 * torch.randn((4 * size, guess_mod.DIN), generator=gen, device="cuda"))
            perm = torch.randperm(4 * size, generator=gen, device="cuda")
            sets.append((trainer.normalize(t, raw.contiguous()), trainer.norm_targets(t, y[pick].contiguous()), perm))
        return {"kind": kind, "trainer": trainer, "sets": sets, "rows": size}
    raise ValueError(kind)


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "single_point":
        ctx = ScfContext(state["nat"], state["xyz"])
        ctx.hcore()
        r = ctx.run()
        p = ctx.density()
        ctx.close()
        return {"escf": r.escf, "p": p}
    if kind == "scf":
        ctx = state["ctx"]
        if state["mode"] == "plain":
            r = ctx.run()
        elif state["mode"] == "pulay":
            r = ctx.run(pseudo=True, pulay=True)
        else:
            ctx.learned_guess(state["model"])
            r = ctx.run(pseudo=True, precision=1, pulay=True, guess=True, shift=0.0)
        return {"escf": r.escf, "p": state["p"], "eigs": state["eigs"]}
    if kind == "batch":
        escf, _, converged, _ = state["batch"].run()
        return {"escf": escf, "converged": converged}
    if kind == "mozyme":
        occ = mozyme.Lmos(state["layout"], state["occ"])
        vir = mozyme.Lmos(state["layout"], state["vir"])
        r = mozyme.scf_run(state["layout"], occ, vir, state["coord"], state["w"], state["h"], state["enuclr"],
                           state["atheat"])
        occ.close()
        vir.close()
        return {"escf": r["escf"], "p": r["p"], "f": r["f"]}
    if kind == "fock":
        kernels.fock2(state["atoms"], state["f"], state["h"], state["p"], state["pa"], state["w"])
        return state["f"]
    if kind == "diagonalise":
        c, eigs = kernels.eigh_packed(state["f"].clone())  # the solver perturbs its argument's diagonal
        return {"eigs": eigs, "p": kernels.density(c, state["nocc"])}
    if kind == "pseudo_step":
        c = state["c"].clone()                              # rotated in place
        kernels.pseudo_diag(state["f"], c, state["eigs"], state["nocc"])
        return {"c": c, "p": kernels.density(c.T, state["nocc"])}
    if kind == "gradient":
        return state["ctx"].gradient()
    if kind == "train":
        trainer, rows = state["trainer"], state["rows"]
        for t, (x, y, perm) in enumerate(state["sets"]):
            for s in range(4):
                idx = perm[s * rows:(s + 1) * rows]
                trainer.step(t, x[idx], y[idx], 1.0e-3)
        return trainer.get()[0]
    raise ValueError(kind)


# -------------------------------------------------------------- least work
def _n2elec(heavy, light):
    """Packed two-electron integrals of a system with that many sp and s atoms."""
    return 50.0 * heavy * (heavy + 1) + 10.0 * heavy * light + 0.5 * light * (light + 1)


def _iteration_flops(n, nocc, n2, full):
    """One SCF iteration: the Fock build over the integrals, the eigensolve
    (reduction and back-transformation of the occupied vectors) or the Fmo
    product and rotations, and the density."""
    diag = 4.0 * n ** 3 / 3.0 + 2.0 * n * n * nocc if full else \
        2.0 * n * n * nocc + 2.0 * n * nocc * (n - nocc) + 6.0 * n * nocc * (n - nocc)
    return 8.0 * n2 + diag + n * n * nocc


def work(case):
    kind, size = case["kind"], case.get("size")
    if kind == "train":
        rows = 20.0 * size
        weights = guess_mod.NTYPES * guess_mod.PER_TYPE
        per_row = 2.0 * (guess_mod.DIN * 128 + 2 * 128 * 128 + 128 * guess_mod.DOUT)
        return {"bytes": rows * (2.0 * guess_mod.DIN + 4.0 * guess_mod.DOUT) + 8.0 * weights,
                "flops": 3.0 * per_row * rows}
    if kind == "batch":
        nbytes = flops = 0.0
        for c in (3 + k % 18 for k in range(size)):
            n, n2 = 6 * c + 2, _n2elec(c, 2 * c + 2)
            nbytes += 8.0 * (n2 + n * (n + 1) / 2)
            flops += 10.0 * _iteration_flops(n, 3 * c + 1, n2, True)
        return {"bytes": nbytes, "flops": flops}
    if kind == "single_point":
        c, w = case["carbons"], case["waters"]
        hydrogens = (2 * c + 2 if c else 0) + 2 * w
        n, nocc = 4 * (c + w) + hydrogens, (3 * c + 1 if c else 0) + 4 * w
        return {"bytes": 8.0 * n * (n + 1) / 2,
                "flops": 12.0 * _iteration_flops(n, nocc, _n2elec(c + w, hydrogens), True)}
    n = size if kind == "diagonalise" else 6 * size
    nocc, mpack, n2 = 2 * n // 3, n * (n + 1) / 2, _n2elec(size, 2 * size)
    if kind == "scf":
        full, pseudo = {"plain": (13.0, 0.0), "pulay": (3.0, 12.0), "fast": (2.0, 15.0)}[case["mode"]]
        pulay = 2.0 * n ** 3 if pseudo else 0.0
        return {"bytes": 8.0 * (n2 + 2.0 * mpack + n),
                "flops": full * _iteration_flops(n, nocc, n2, True) +
                pseudo * (_iteration_flops(n, nocc, n2, False) + pulay)}
    if kind == "mozyme":
        # stored pairs within the cutoff: about 100 waters around each
        near = min(size, 100)
        n2s = 50.0 * size * near + 10.0 * size * 2 * near + 2.0 * size * near
        return {"bytes": 8.0 * (n2s + 3.0 * 18.0 * size * near), "flops": 20.0 * 8.0 * n2s}
    if kind == "fock":
        return {"bytes": 8.0 * (n2 + 4.0 * mpack), "flops": 8.0 * n2}
    if kind == "diagonalise":
        return {"bytes": 8.0 * (2.0 * mpack + n), "flops": 4.0 * n ** 3 / 3.0 + 2.0 * n * n * nocc + n * n * nocc}
    if kind == "pseudo_step":
        return {"bytes": 8.0 * (2.0 * mpack + 2.0 * n * n + n),
                "flops": _iteration_flops(n, nocc, 0.0, False)}
    if kind == "gradient":
        pairs = 1.5 * size * (3.0 * size - 1.0)
        # four evaluations of a pair's integrals and energy, of the order of 1000 operations
        return {"bytes": 8.0 * (mpack + 6.0 * 3 * size), "flops": 4000.0 * pairs}
    raise ValueError(kind)


# ----------------------------------------------------------- 64-bit results
def _exact_fock(state):
    """F = H + G(P) in 64 bits by contraction over the pair blocks of W."""
    nat = state["ctx"].nat
    p = _full(state["p"], state["ctx"].norbs)
    f = _full(state["h"], state["ctx"].norbs)
    w = state["w"]
    nor = _orbitals(nat)
    lim = nor * (nor + 1) // 2
    first = np.cumsum(nor) - nor
    cum = np.cumsum(lim) - lim
    row = np.cumsum(lim * (cum + lim)) - lim * (cum + lim)
    pair = np.array([[max(i, j) * (max(i, j) + 1) // 2 + min(i, j) for j in range(4)] for i in range(4)])
    dev = p.device
    for na in (1, 4):
        for nb in (1, 4):
            la, lb = na * (na + 1) // 2, nb * (nb + 1) // 2
            a_of, b_of = np.nonzero((nor[:, None] == na) & (nor[None, :] == nb) &
                                    (np.arange(len(nat))[None, :] <= np.arange(len(nat))[:, None]))
            for s in range(0, len(a_of), 20000):
                a, b = a_of[s:s + 20000], b_of[s:s + 20000]
                off = torch.from_numpy(row[a] + lim[a] * cum[b]).to(dev)
                blk = w[off[:, None] + torch.arange(la * lb, device=dev)].view(-1, la, lb)
                pa = torch.from_numpy(pair[:na, :na]).to(dev)
                pb = torch.from_numpy(pair[:nb, :nb]).to(dev)
                full = blk[:, pa][:, :, :, pb]               # (pairs, na, na, nb, nb): (mu nu | lam sig)
                ia = torch.from_numpy(first[a][:, None] + np.arange(na)).to(dev)
                ib = torch.from_numpy(first[b][:, None] + np.arange(nb)).to(dev)
                same = torch.from_numpy(a == b).to(dev)
                daa = p[ia[:, :, None], ia[:, None, :]]
                dbb = p[ib[:, :, None], ib[:, None, :]]
                dab = p[ia[:, :, None], ib[:, None, :]]
                f.index_put_((ia[:, :, None], ia[:, None, :]), torch.einsum("zmnls,zls->zmn", full, dbb), True)
                other = torch.einsum("zmnls,zmn->zls", full, daa)
                other[same] = 0.0
                f.index_put_((ib[:, :, None], ib[:, None, :]), other, True)
                exch = -0.5 * torch.einsum("zmnls,zns->zml", full, dab)
                f.index_put_((ia[:, :, None], ib[:, None, :]), exch, True)
                mirror = exch.transpose(1, 2).clone()
                mirror[same] = 0.0
                f.index_put_((ib[:, :, None], ia[:, None, :]), mirror, True)
    i, j = torch.tril_indices(f.shape[0], f.shape[0], device=dev)
    return f[i, j]


def exact(case, seed):
    if case["kind"] == "fock":
        return _exact_fock(prepare(case, seed))
    if case["kind"] == "diagonalise":
        state = prepare(case, seed)
        n = case["size"]
        a = _full(state["f"], n)
        a += torch.diag(1.0e-10 * torch.arange(1, n + 1, dtype=torch.float64, device="cuda"))
        eigs, c = torch.linalg.eigh(a)
        p = 2.0 * c[:, :state["nocc"]] @ c[:, :state["nocc"]].T
        i, j = torch.tril_indices(n, n, device="cuda")
        return {"eigs": eigs, "p": p[i, j]}
    return None
