"""Performance cases of the template matcher: what its users have it do.

Three kinds of call, each through a public entry point:

``objects``   `Jess.query` / `Jess.query_arrays` on `Molecule` and `Template`
              objects, as a PyJess program calls them: every call packs and
              uploads its molecules, searches them and copies the hits out.
``resident``  the C ABI (``include/pjg.h``, through its ctypes binding) with
              the template and structure handles kept, as a service does that
              searches one structure set again and again: `pjg_query`, then
              `pjg_results_copy`.
``rows``      `pjg_superpose_noalloc` on device buffers.

Structures and templates come from `pyjess_gb300.workloads` (the generators
of the benchmark configurations), drawn from the seed.
"""

import ctypes
import math

import numpy as np
import torch

from pyjess_gb300 import Jess, Molecule, Template, TemplateAtom, _native
from pyjess_gb300 import workloads as W
from pyjess_gb300._abi import QueryParams

_COMMON = {"rmsd": 2.0, "cutoff": 1.5, "dynamic": 1.5, "best": False, "max_candidates": -1, "ignore": "none",
           "reorder": True, "precision": "fp32", "dense": False, "large": 0.0, "lo": 0, "hi": 0, "tlo": 2, "thi": 8}


def _case(**kw):
    return {**_COMMON, **kw}


def listed():
    return [
        # one active-site template tried on one small protein, hits iterated:
        # the smallest call there is (an interactive session, a unit of a loop)
        _case(name="one_template", kind="objects", iterate=True, structures=1, lo=300, hi=300, templates=1, tlo=3,
              thi=3),
        # one mid-sized protein against a family's templates
        _case(name="one_protein_200", kind="objects", iterate=False, structures=1, lo=1000, hi=1000, templates=200,
              tlo=3, thi=6),
        # annotating one protein with a whole template library: the best hit
        # of each template
        _case(name="annotate_3000", kind="objects", iterate=False, structures=1, lo=420, hi=420, templates=3000,
              best=True),
        # screening a structure collection with a few new templates; the
        # collection stays on the device
        _case(name="screen_1200x3", kind="resident", structures=1200, templates=3, tlo=3, thi=5),
        # a batch of proteins against a library, every hit as columns, the
        # superposed atoms with them
        _case(name="batch_97x2001", kind="objects", iterate=False, structures=97, templates=2001, transform=True),
        # FP64 distance tests throughout, chains ignored between residues
        _case(name="fp64_61x1003", kind="resident", structures=61, templates=1003, precision="fp64",
              ignore="residues"),
        # the first candidates of each template only, in the template's own
        # atom order, chains ignored altogether (flexible geometry: 2 A)
        _case(name="first_ten_53x601", kind="resident", structures=53, templates=601, max_candidates=10,
              ignore="atoms", reorder=False, cutoff=2.0, dynamic=2.0),
        # templates of 33 to 42 atoms (extended sites) among ordinary ones
        _case(name="large_sites_24x120", kind="objects", iterate=False, structures=24, lo=200, hi=600,
              templates=120, large=0.2),
        # backbone templates that any residue matches, large structures: the
        # best hit of each pair among up to 10,000 candidates
        _case(name="dense_best_8x48", kind="resident", structures=8, lo=2000, hi=5000, templates=48, tlo=2, thi=3,
              dense=True, best=True, max_candidates=10000, rmsd=3.0, cutoff=3.0, dynamic=3.0),
        # the same templates, every hit of small structures
        _case(name="dense_all_5x12", kind="resident", structures=5, lo=300, hi=500, templates=12, tlo=2, thi=3,
              dense=True, max_candidates=50, rmsd=3.0, cutoff=3.0, dynamic=3.0),
        # a structure database against a template library: the largest job
        _case(name="database_1000x4000", kind="resident", structures=1000, templates=4000),
        # superposing candidate assignments that the caller found itself
        _case(name="superpose_rows", kind="rows", rows=300000, atoms=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    u = rng.random()
    if u < 0.15:
        return _case(kind="rows", rows=_log_int(rng, 500, 1 << 20), atoms=rng.randint(3, 32))
    if u < 0.25:
        best = rng.random() < 0.5
        lo = _log_int(rng, 150, 2000 if best else 400)
        return _case(kind="resident", structures=rng.randint(1, 6), lo=lo, hi=lo + lo // 3,
                     templates=rng.randint(1, 24 if best else 12), tlo=2, thi=3, dense=True, best=best,
                     max_candidates=_log_int(rng, 10, 10000) if best else rng.randint(5, 50), rmsd=3.0, cutoff=3.0,
                     dynamic=3.0)
    kind = "objects" if rng.random() < 0.5 else "resident"
    structures = _log_int(rng, 1, 100 if kind == "objects" else 1000)
    templates = _log_int(rng, 1, 3000)
    while structures * templates > 1500000:
        templates = _log_int(rng, 1, 3000)
    reach = rng.choice([1.0, 1.5, 1.5, 2.0])
    case = _case(kind=kind, structures=structures, templates=templates, cutoff=reach, dynamic=reach,
                 best=rng.random() < 0.3, ignore=rng.choice(["none", "none", "residues", "atoms"]),
                 reorder=rng.random() < 0.8, precision="fp64" if rng.random() < 0.15 else "fp32",
                 max_candidates=rng.choice([-1, -1, -1, 1, 25, 1000]),
                 large=0.1 if structures * templates < 5000 and rng.random() < 0.2 else 0.0)
    if kind == "objects":
        case["iterate"] = structures == 1 and templates <= 10 and reach < 2
    return case


# --- inputs -----------------------------------------------------------------


def _inputs(case, seed):
    """(structures, template specs) of a case, from the seed alone."""
    ns, nt = case["structures"], case["templates"]
    kids = np.random.SeedSequence([20261205, seed]).spawn(ns + nt + 1)
    meta = np.random.Generator(np.random.PCG64(kids[-1]))
    if case["lo"]:
        lengths = meta.integers(case["lo"], case["hi"] + 1, size=ns)
    else:  # chain lengths of a structure database
        lengths = np.clip(np.round(np.exp(np.log(350) + 0.6 * meta.normal(size=ns))), 80, 3000).astype(int)
    structs = W.make_structures([np.random.Generator(np.random.PCG64(k)) for k in kids[:ns]], lengths,
                                meta.integers(1, 5, size=ns))
    sizes = np.arange(case["tlo"], case["thi"] + 1)
    odds = sizes.astype(float) ** -2.0
    specs = []
    for j in range(nt):
        rng = np.random.Generator(np.random.PCG64(kids[ns + j]))
        donor = structs[int(meta.integers(ns))]
        if meta.random() < case["large"]:
            specs.append(W.make_template(rng, donor, int(rng.integers(11, 15)), radius=14.0))
        elif case["dense"]:
            specs.append(W.make_template(rng, donor, int(meta.choice(sizes)), permissive=True, atoms_per_res=2))
        else:
            specs.append(W.make_template(rng, donor, int(meta.choice(sizes, p=odds / odds.sum()))))
    return structs, specs


def _token(raw):
    return raw.split(b"\0")[0].replace(b"_", b"").decode()


def _molecule(s, index):
    """The structure as a `Molecule`, read from PDB text."""
    lines = []
    for (x, y, z), name, res, chain, seq, serial in zip(s["xyz"].tolist(), s["name"], s["resname"], s["chain"],
                                                        s["res_seq"].tolist(), s["serial"].tolist()):
        nm = _token(name.tobytes())
        lines.append(f"ATOM  {serial % 100000:5d}  {nm:<3s} {_token(res.tobytes()):3s} {chr(chain[1])}{seq:4d}    "
                     f"{x:8.3f}{y:8.3f}{z:8.3f}  1.00  0.00           {nm[0]}  ")
    return Molecule.loads("\n".join(lines) + "\nEND\n", id=f"m{index}")


def _template(spec, index):
    return Template([TemplateAtom(chain_id=ch.decode().strip(), residue_number=rs, x=float(p[0]), y=float(p[1]),
                                  z=float(p[2]), residue_names=[_token(r) for r in rn],
                                  atom_names=[_token(n) for n in nm], distance_weight=w, match_mode=int(code))
                     for code, rs, ch, p, w, nm, rn in zip(spec.code, spec.res_seq, spec.chain, spec.xyz,
                                                           spec.weight, spec.names, spec.resnames)], id=f"t{index}")


def _rows(case, seed):
    """Candidate assignments near a template: rigid motions of it with noise."""
    n, m = case["atoms"], case["rows"]
    g = np.random.Generator(np.random.PCG64(np.random.SeedSequence([20261206, seed])))
    tpl = g.normal(scale=4.0, size=(n, 3)) + 20.0
    q = g.normal(size=(m, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, x, y, z = q.T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                  2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                  2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(m, 3, 3)
    mol = np.einsum("mij,nj->mni", R, tpl - tpl.mean(0)) + g.normal(scale=30.0, size=(m, 1, 3))
    mol += g.normal(size=(m, n, 3)) * g.uniform(0.05, 2.0, size=(m, 1, 1))
    return mol, tpl


# hits that an iterated query's caller keeps (at most 20 templates, one molecule)
_ITERATED = 4000


class _State:
    pass


_FIELDS = (("structure", np.int32, ()), ("template", np.int32, ()), ("ordinal", np.int64, ()),
           ("rmsd", np.float64, ()), ("rotation", np.float64, (9,)), ("centres", np.float64, (6,)),
           ("atom_offset", np.int64, ()), ("atoms", np.int32, ()))


def _room(case):
    """Hits and hit atoms that the caller's columns have room for: well above
    what the generators' workloads give (a template finds its donor many times
    over, so the few-structure cases need more a pair)."""
    ns, nt = case["structures"], case["templates"]
    if case["best"]:
        hits = ns * nt
    elif case["dense"]:
        hits = ns * nt * 60 * max(case["hi"], 400) + 150000
    else:
        pair, donor = {1.0: (0.6, 40), 1.5: (1.6, 100), 2.0: (20, 400)}[case["cutoff"]]
        hits = int(ns * nt * pair) + nt * donor
    most = 6 if case["dense"] else 42 if case["large"] else 3 * case["thi"]
    return hits, hits * (most if case["dense"] or nt < 200 else 12)


def _columns(case):
    """The caller's columns for the hits, zeroed: rows past the last hit stay 0."""
    hits, atoms = _room(case)
    out = {}
    for name, dtype, width in _FIELDS:
        rows = atoms if name == "atoms" else hits + 1 if name == "atom_offset" else hits
        out[name] = np.empty((rows, *width), dtype)
        out[name].fill(0)
    return out


def prepare(case, seed):
    st = _State()
    st.case = case
    if case["kind"] == "rows":
        mol, tpl = _rows(case, seed)
        m = case["rows"]
        st.lib = _native.init()
        st.lib.pjg_superpose_noalloc.argtypes = [ctypes.c_void_p] * 2 + [ctypes.c_int32] * 2 + \
            [ctypes.c_double] + [ctypes.c_void_p] * 6
        st.mol = torch.from_numpy(mol).cuda()
        st.tpl = torch.from_numpy(tpl).cuda()
        new = lambda *shape, dtype=torch.float64: torch.zeros(shape, dtype=dtype, device="cuda")
        st.out = [new(m), new(m, 9), new(m, 6), new(m, dtype=torch.int32), new(1, dtype=torch.int32)]
        return st
    structs, specs = _inputs(case, seed)
    if case["kind"] == "objects":
        st.molecules = [_molecule(s, i) for i, s in enumerate(structs)]
        st.jess = Jess([_template(sp, i) for i, sp in enumerate(specs)])
        st.args = (case["rmsd"], case["cutoff"], case["dynamic"])
        st.options = dict(max_candidates=None if case["max_candidates"] < 0 else case["max_candidates"],
                          ignore_chain=None if case["ignore"] == "none" else case["ignore"],
                          best_match=case["best"], reorder=case["reorder"])
        if not case["iterate"]:
            st.options["precision"] = case["precision"]
            st.out = _columns(case)
            if case.get("transform"):
                st.out["superposed"] = np.zeros((len(st.out["atoms"]), 3))
        return st
    st.templates = _native.Templates(W.pack_templates(specs))
    st.structures = _native.Structures(W.pack(structs))
    st.params = QueryParams(
        rmsd_threshold=case["rmsd"], distance_cutoff=case["cutoff"], max_dynamic_distance=case["dynamic"],
        max_candidates=case["max_candidates"], ignore_chain=("none", "residues", "atoms").index(case["ignore"]),
        best_match=int(case["best"]), reorder=int(case["reorder"]),
        mode=_native.MODE_BATCHED_FP64 if case["precision"] == "fp64" else _native.MODE_BATCHED_FP32)
    st.out = _columns(case)
    st.lib = _native.load()
    return st


def run(state):
    kind = state.case["kind"]
    if kind == "rows":
        rmsd, rot, cen, rows, count = state.out
        status = state.lib.pjg_superpose_noalloc(
            state.mol.data_ptr(), state.tpl.data_ptr(), state.case["rows"], state.case["atoms"], state.case["rmsd"],
            rmsd.data_ptr(), rot.data_ptr(), cen.data_ptr(), rows.data_ptr(), count.data_ptr(),
            torch.cuda.current_stream().cuda_stream)
        if status:
            raise RuntimeError("pjg_superpose_noalloc")
        return {"rmsd": rmsd, "rotation": rot, "centres": cen, "rows": rows, "count": count}
    if kind == "objects":
        if state.case["iterate"]:
            hits = list(state.jess.query(state.molecules[0], *state.args, **state.options))
            rmsd, transformation, serials = np.zeros(_ITERATED), np.zeros((_ITERATED, 4, 4)), []
            for i, h in enumerate(hits):
                rmsd[i] = h.rmsd
                transformation[i] = h.transformation
                serials += [a.serial for a in h.atoms(transform=False)]
            return {"count": len(hits), "rmsd": rmsd, "transformation": transformation,
                    "serials": np.array(serials + [0] * (24 * _ITERATED - len(serials)))}
        h = state.jess.query_arrays(state.molecules, *state.args, **state.options)
        found = {"structure": h.molecule, "template": h.template, "ordinal": h.ordinal, "rmsd": h.rmsd,
                 "rotation": h.rotation.reshape(-1, 9), "centres": h.centres.reshape(-1, 6),
                 "atom_offset": h.atom_offset, "atoms": h.atoms}
        if state.case.get("transform"):
            found["superposed"] = h.superposed_atoms()
        for name, v in found.items():
            state.out[name][:len(v)] = v
        return {"count": len(h), **state.out}
    result = _native.query(state.templates, state.structures, state.params)
    count, atoms = state.lib.pjg_results_count(result.handle), state.lib.pjg_results_atom_count(result.handle)
    if count > len(state.out["rmsd"]) or atoms > len(state.out["atoms"]):
        raise RuntimeError(f"{count} hits with {atoms} atoms: more than there is room for")
    status = state.lib.pjg_results_copy(result.handle, *(state.out[name].ctypes.data for name, _, _ in _FIELDS))
    if status:
        raise RuntimeError("pjg_results_copy")
    return {"count": count, **state.out}


def work(case):
    """Inputs read once and hits written once.  A residue has 7.9 atoms of 42
    bytes, a template residue three atoms of 60; a hit has 148 bytes and four
    an atom.  Hits a pair (which only the search tells) are what the
    generators' workloads give on average.  Operations: the superposition of
    each hit (its covariance, the 4 x 4 eigenproblem)."""
    if case["kind"] == "rows":
        m, n = case["rows"], case["atoms"]
        return {"bytes": m * (24 * n + 8 + 72 + 48 + 4) + 24 * n, "flops": m * (33 * n + 400)}
    residues = (case["lo"] + case["hi"]) / 2 if case["lo"] else 420
    pairs = case["structures"] * case["templates"]
    if case["dense"]:
        atoms, hits = 5, pairs * (1 if case["best"] else 8000)
    else:
        sizes = range(case["tlo"], case["thi"] + 1)
        atoms = 3 * sum(k ** -1 for k in sizes) / sum(k ** -2 for k in sizes)
        hits = pairs * (0.14 if case["best"] else 1.2)
    data = case["structures"] * residues * 7.9 * 42 + case["templates"] * atoms * 60
    return {"bytes": int(data + hits * (148 + 4 * atoms)), "flops": int(hits * (33 * atoms + 400))}


# --- the same results in plain numpy, 64 bits --------------------------------
#
# The search as the reference describes it: a candidate list per template atom
# (residue names in the template's order, then serial), a kd-tree per list
# (median of three, Lomuto partition, axes cycling, right subtree reported
# first), levels by list length, depth first.

_PARTNERS = [("ASP", "OD1", "OD2"), ("GLU", "OE1", "OE2"), ("ASN", "OD1", "ND2"), ("GLN", "OE1", "NE2"),
             ("ARG", "NH1", "NH2"), ("HIS", "ND1", "CD2"), ("HIS", "CE1", "NE2"), ("PHE", "CD1", "CD2"),
             ("PHE", "CE1", "CE2"), ("TYR", "CD1", "CD2"), ("TYR", "CE1", "CE2"), ("LEU", "CD1", "CD2"),
             ("VAL", "CG1", "CG2")]
_PARTNER = {(r, x): y for r, a, b in _PARTNERS for x, y in ((a, b), (b, a))}


def _kd_order(x):
    perm = list(range(len(x)))
    stack = [(0, len(x), 0)]
    while stack:
        lo, n, axis = stack.pop()
        if n <= 1:
            continue
        key = x[:, axis]
        left, right, k = lo, lo + n - 1, lo + n // 2
        while left != right:
            mid = (left + right - 2 * lo + 1) // 2 + lo
            l, r, m = key[perm[left]], key[perm[right]], key[perm[mid]]
            p = left if (l > m) != (l > r) else mid if (m < l) != (m < r) else right
            perm[right], perm[p] = perm[p], perm[right]
            pivot, store = key[perm[right]], left
            for i in range(left, right):
                if key[perm[i]] <= pivot:
                    perm[i], perm[store] = perm[store], perm[i]
                    store += 1
            perm[store], perm[right] = perm[right], perm[store]
            if store == k:
                break
            left, right = (left, store - 1) if k < store else (store + 1, right)
        stack.append((lo, n // 2, (axis + 1) % 3))
        stack.append((lo + n // 2, n - n // 2, (axis + 1) % 3))
    return perm[::-1]


def _superpose(a, b):
    """Least-squares fits of rows a (m, n, 3) onto b: rmsd, rotation, centres."""
    ca, cb = a.mean(1), b.mean(1)
    p, q = a - ca[:, None], b - cb[:, None]
    u, _, vt = np.linalg.svd(np.einsum("mni,mnj->mij", q, p))
    sign = np.ones((len(a), 3))
    sign[:, 2] = np.sign(np.linalg.det(u) * np.linalg.det(vt))
    R = np.einsum("mij,mj,mjk->mik", u, sign, vt)
    left = q - np.einsum("mij,mnj->mni", R, p)
    return np.sqrt((left ** 2).sum((1, 2)) / a.shape[1]), R, np.stack([ca, cb], 1)


def _search_pair(s, spec, case, cache):
    n = len(spec.code)
    xyz, seq, chain = s["xyz"], s["res_seq"], s["chain"][:, 1].astype(int)
    lists = []
    for k in range(n):
        names = [_token(v) for v in spec.names[k]]
        want = []
        for r in (_token(v) for v in spec.resnames[k]):
            if r not in want:
                want.append(r)
        key = (spec.code[k], tuple(names), tuple(want))
        if key not in cache:
            found = []
            for r in want:
                for a in cache["residues"].get(r, ()):
                    nm = cache["names"][a]
                    if nm in names or (spec.code[k] == 1 and _PARTNER.get((r, nm)) in names) or \
                            (spec.code[k] == 3 and any((("_" + nm + "__")[:2] if len(nm) < 4 else nm[:2]) ==
                                                       (("_" + v + "__")[:2] if len(v) < 4 else v[:2])
                                                       for v in names)):
                        found.append(a)
            cache[key] = [np.array(found, int), None]
        lists.append(cache[key])
        if len(lists[-1][0]) == 0:
            return []
    order = sorted(range(n), key=lambda k: (len(lists[k][0]), k)) if case["reorder"] else list(range(n))
    pos = np.array(spec.xyz)
    dist = np.sqrt(((pos[:, None] - pos[None]) ** 2).sum(-1))
    tchain = [c[1] for c in spec.chain]
    rows = []

    def visit(level, chosen):
        if level == n:
            row = [0] * n
            for k, a in zip(order, chosen):
                row[k] = a
            rows.append(row)
            return
        k = order[level]
        entry = lists[k]
        if level == 0:
            for a in entry[0]:
                visit(1, [a])
            return
        if entry[1] is None:
            entry[1] = entry[0][_kd_order(xyz[entry[0]])]
        c = entry[1]
        ok = np.ones(len(c), bool)
        for j, a in zip(order, chosen):
            reach = min(case["cutoff"] + spec.weight[j] + spec.weight[k], case["dynamic"])
            lo, hi = max(dist[j, k] - reach, 0.5), dist[j, k] + reach
            v = xyz[a] - xyz[c]
            d2 = v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1] + v[:, 2] * v[:, 2]
            ok &= ~((d2 < lo * lo) | (d2 > hi * hi))
            same = chain[c] == chain[a]
            near = seq[c] == seq[a]
            rule = near == (spec.res_seq[j] == spec.res_seq[k])
            if case["ignore"] == "none":
                rule = np.where(same, rule, True) & (same == (tchain[j] == tchain[k]))
            elif case["ignore"] == "residues":
                rule &= ~(near & ~same)
            ok &= rule
        for a in c[ok]:
            visit(level + 1, chosen + [a])

    visit(0, [])
    return rows


def exact(case, seed):
    if case["kind"] == "rows":
        mol, tpl = _rows(case, seed)
        rmsd, R, centres = _superpose(mol, np.broadcast_to(tpl, mol.shape))
        return {"rmsd": rmsd, "rotation": R.reshape(-1, 9), "centres": centres.reshape(-1, 6), "rows": None,
                "count": None}
    # larger searches take plain Python too long; cut streams and best hits are
    # compared with the listed cases that take every hit
    if case["structures"] * case["templates"] > 250 or case["dense"] or case["large"] or case["max_candidates"] >= 0 \
            or case["best"] or case["cutoff"] > 1.5:
        return None
    structs, specs = _inputs(case, seed)
    found = []
    for i, s in enumerate(structs):
        names = [_token(v.tobytes()) for v in s["name"]]
        residues = {}
        for a, r in enumerate(s["resname"]):
            residues.setdefault(_token(r.tobytes()), []).append(a)
        cache = {"names": names, "residues": residues}
        if case["kind"] == "objects":
            s = {**s, "xyz": np.round(s["xyz"], 3)}
        for t in reversed(range(len(specs))):
            rows = _search_pair(s, specs[t], case, cache)
            if not rows:
                continue
            at = np.array(rows)
            b = np.broadcast_to(np.array(specs[t].xyz), at.shape + (3,))
            rmsd, R, centres = _superpose(s["xyz"][at], b)
            keep = rmsd <= case["rmsd"]
            found.append((i, t, np.flatnonzero(keep), rmsd[keep], R[keep], centres[keep], at[keep]))
    cat = lambda q, shape: np.concatenate([f[q] for f in found]) if found else np.zeros(shape)
    rmsd, R, centres = cat(3, 0), cat(4, (0, 3, 3)), cat(5, (0, 2, 3))
    pad = lambda v, rows: np.concatenate([v, np.zeros((rows - len(v), *v.shape[1:]))])
    if case.get("iterate"):
        T = np.zeros((len(rmsd), 4, 4))
        T[:, 3, 3] = 1
        T[:, :3, :3] = R
        T[:, :3, 3] = centres[:, 1] - np.einsum("mij,mj->mi", R, centres[:, 0])
        return {"count": None, "rmsd": pad(rmsd, _ITERATED), "transformation": pad(T, _ITERATED), "serials": None}
    rows = _room(case)[0]
    out = {"count": None, **{name: None for name, _, _ in _FIELDS}, "rmsd": pad(rmsd, rows),
           "rotation": pad(R.reshape(-1, 9), rows), "centres": pad(centres.reshape(-1, 6), rows)}
    if case.get("transform"):
        out["superposed"] = None
    return out
