"""The order-free search (k_search_free, k_unit_order) against the oracle.

Each test drives a path of it: residues that are not contiguous in the file
or share their number, pairs searched in items of seeds, entries spilled to a
later launch, units of one row up to tens of thousands, structures with more
atom kinds than it takes (searched in order), and the pairs' streams cut by
max_candidates.  Bar as in test_gpu_parity.py: identical ordered hits,
warnings and search counters, RMSD within RMSD_TOL.
"""

import numpy as np
import pytest

from test_gpu_parity import compare, gpu_query
from helpers import hit_keys

pytestmark = pytest.mark.gpu

PARAMS = dict(rmsd_threshold=2.0, distance_cutoff=1.5, max_dynamic_distance=1.5)


def _structures(seed, lengths, chains=2):
    from pyjess_gb300 import workloads as W

    return W.make_structures([np.random.default_rng([seed, i]) for i in range(len(lengths))], lengths,
                             [chains] * len(lengths))


def _templates(seed, structs, n, lo=2, hi=7, **kw):
    from pyjess_gb300 import workloads as W

    rng = np.random.default_rng([seed, 99])
    return [W.make_template(rng, structs[int(rng.integers(len(structs)))], int(rng.integers(lo, hi)), **kw)
            for _ in range(n)]


@pytest.mark.parametrize("ignore", [0, 1, 2])
@pytest.mark.parametrize("mode", ["fp32", "fp64"])
def test_scattered_residues(mode, ignore):
    """Atoms in random file order, residue numbers that repeat within and
    across chains and go below zero: the atoms of a residue are found by key
    (or by number alone), wherever they stand."""
    from pyjess_gb300 import workloads as W

    structs = _structures(31, [33, 130, 270, 310])
    specs = _templates(31, structs, 60)
    rng = np.random.default_rng(7)
    for s in structs:
        s["res_seq"] = ((s["res_seq"] * 7) % 90 - 12).astype(np.int32)
        order = rng.permutation(len(s["xyz"]))
        for k in ("xyz", "name", "resname", "res_seq", "chain", "serial"):
            s[k] = np.ascontiguousarray(s[k][order])
    _, ref = compare(W.pack_templates(specs), W.pack(structs), mode=mode, ignore_chain=ignore, **PARAMS)
    assert ref["hits"]["count"] > 0


@pytest.mark.parametrize("ignore", [0, 2])
def test_fp64_mode_near_annulus_bounds(ignore):
    """Atoms within 1e-6 A of annulus boundaries in FP64 mode, whose annuli
    hold no FP32 bounds to reject a point with: the oracle's hits."""
    from pyjess_gb300 import workloads as W

    wl = W.config(3, n_structures=20, n_templates=200)
    res, ref = compare(wl.templates, wl.structures, mode="fp64", ignore_chain=ignore, **wl.params)
    assert ref["hits"]["count"] > 0 and res.stats()["fp64_rechecks"] == 0


@pytest.mark.parametrize("kw", [dict(), dict(best_match=True), dict(max_candidates=0), dict(max_candidates=5),
                                dict(max_candidates=300), dict(best_match=True, max_candidates=7),
                                dict(reorder=False), dict(reorder=False, max_candidates=40)])
def test_pairs_in_items(kw):
    """Structures whose lists exceed the first instance's frontier, 2.2 A of
    play: pairs in items of seeds, units from one row to hundreds, streams cut
    in the middle."""
    from pyjess_gb300 import workloads as W

    structs = _structures(32, [900, 1500, 60])
    specs = _templates(32, structs, 24, hi=5)
    _, ref = compare(W.pack_templates(specs), W.pack(structs), rmsd_threshold=1.6, distance_cutoff=2.2,
                     max_dynamic_distance=2.2, **kw)
    assert ref["hits"]["count"] > 0


@pytest.mark.parametrize("mode", ["fp32", "fp64"])
@pytest.mark.parametrize("kw", [dict(), dict(max_candidates=20), dict(best_match=True, max_candidates=1000)])
def test_spilled_entries(mode, kw):
    """Element-matched templates with 2 A of play in small structures: a few
    seeds with 100,000 and more partial assignments, so entries are spilled
    to later launches and a unit has up to 70,000 rows."""
    from pyjess_gb300 import workloads as W

    for seed in (7, 8):
        rng = np.random.default_rng(seed)
        structs = W.make_structures([rng], [60], [1])
        specs = [W.make_template(rng, structs[0], 6, modes=(3,), mode_p=(1.0,)) for _ in range(2)]
        compare(W.pack_templates(specs), W.pack(structs), mode=mode, rmsd_threshold=2.0, distance_cutoff=2.0,
                max_dynamic_distance=2.0, **kw)


@pytest.mark.parametrize("residues", [1, 2])
@pytest.mark.parametrize("kw", [dict(), dict(max_candidates=3), dict(best_match=True),
                                dict(best_match=True, max_candidates=20)])
def test_templates_of_one_and_two_atoms(monkeypatch, residues, kw):
    """One atom (left to the search in order) and two (every rotation
    undefined: all rows warn), with streams longer than a thread takes: the
    warnings of the search in order (PJG_LEAF_LEVELS)."""
    from pyjess_gb300 import workloads as W

    structs = _structures(33, [150, 400])
    specs = _templates(33, structs, 12, lo=residues, hi=residues + 1, atoms_per_res=1)
    pt, ps = W.pack_templates(specs), W.pack(structs)
    free = gpu_query(pt, ps, **PARAMS, **kw)
    monkeypatch.setenv("PJG_LEAF_LEVELS", "4")
    ordered = gpu_query(pt, ps, **PARAMS, **kw)
    assert hit_keys(free.arrays()) == hit_keys(ordered.arrays())
    a, b = free.warnings(), ordered.warnings()
    assert len(a[0]) > 0 and np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("kinds", [31, 33, 1023, 1025])
def test_many_atom_kinds(kinds):
    """Distinct (residue, atom) names of a structure around a word of kind
    bits and around the most the order-free search takes."""
    from pyjess_gb300 import workloads as W

    structs = _structures(34, [220, 90])
    specs = _templates(34, structs, 30)
    rng = np.random.default_rng(kinds)
    for s in structs:
        have = len(np.unique(np.concatenate([s["resname"], s["name"]], 1), axis=0))
        if kinds < have:  # keep the most common kinds only
            both = [bytes(v) for v in np.concatenate([s["resname"], s["name"]], 1)]
            names, counts = np.unique(both, return_counts=True)
            keep = np.isin(both, names[np.argsort(-counts, kind="stable")[:kinds]])
            for k in ("xyz", "name", "resname", "res_seq", "chain", "serial"):
                s[k] = np.ascontiguousarray(s[k][keep])
        else:  # ligand atoms of names of their own
            m = kinds - have
            extra = {"xyz": s["xyz"][rng.integers(len(s["xyz"]), size=m)] + rng.normal(scale=3.0, size=(m, 3)),
                     "name": np.frombuffer(b"".join(b"X%03d" % (i % 1000) for i in range(m)), np.uint8).reshape(m, 4),
                     "resname": np.frombuffer(b"".join(b"L%02d\0" % (i // 100) for i in range(m)),
                                              np.uint8).reshape(m, 4),
                     "res_seq": np.arange(900, 900 + m, dtype=np.int32), "chain": np.tile(s["chain"][:1], (m, 1)),
                     "serial": np.arange(9000, 9000 + m, dtype=np.int32)}
            for k, v in extra.items():
                s[k] = np.ascontiguousarray(np.concatenate([s[k], v]))
    _, ref = compare(W.pack_templates(specs), W.pack(structs), **PARAMS)
    assert ref["hits"]["count"] > 0 or kinds < 40


def test_same_as_search_in_order(monkeypatch):
    """The same query with the lists ordered up front (PJG_LEAF_LEVELS): every
    column bit for bit the same."""
    from pyjess_gb300 import workloads as W

    wl = W.config(3, n_structures=40, n_templates=400)
    free = gpu_query(wl.templates, wl.structures, **wl.params)
    monkeypatch.setenv("PJG_LEAF_LEVELS", "4")
    ordered = gpu_query(wl.templates, wl.structures, **wl.params)
    a, b = free.arrays(), ordered.arrays()
    assert hit_keys(a) == hit_keys(b)
    for k in ("rmsd", "rotation", "centres"):
        assert np.array_equal(a[k], b[k]), k
    for k in ("pairs", "candidate_entries", "partials", "complete", "passing", "hits", "fp64_rechecks",
              "bytes_candidates", "bytes_expansion"):
        assert free.stats()[k] == ordered.stats()[k], k


@pytest.mark.parametrize("step", [None, 0.05])
@pytest.mark.parametrize("residues", [31, 32, 33, 65, 511, 512, 513, 2047, 2048, 2049])
def test_rows_told_apart_in_lists_of(residues, step):
    """Backbone templates any residue matches (lists of as many entries as
    residues) around the sizes at which a kd node is taken apart another way,
    without ties and on a 0.05 A grid."""
    from pyjess_gb300 import workloads as W

    structs = _structures(36, [residues])
    if step:
        for s in structs:
            s["xyz"] = np.round(s["xyz"] / step) * step
    specs = _templates(36, structs, 3, lo=2, hi=4, permissive=True)
    reach = 2.5 if residues < 100 else 1.2 if residues < 600 else 0.9
    _, ref = compare(W.pack_templates(specs), W.pack(structs), rmsd_threshold=2.5, distance_cutoff=reach,
                     max_dynamic_distance=reach)
    assert ref["hits"]["count"] > 1


def test_concurrent_queries():
    """Queries from four threads on shared handles (each takes a stream and
    its kept blocks for itself), structure sets made and dropped meanwhile:
    the hits of a query alone."""
    import threading

    from pyjess_gb300 import _native, workloads as W
    from pyjess_gb300._abi import QueryParams

    wl = W.config(3, n_structures=30, n_templates=300)
    T, S = _native.Templates(wl.templates), _native.Structures(wl.structures)
    P = QueryParams(rmsd_threshold=2.0, distance_cutoff=1.5, max_dynamic_distance=1.5, max_candidates=-1,
                    ignore_chain=0, best_match=0, reorder=1, mode=_native.MODE_BATCHED_FP32)
    want = _native.query(T, S, P).arrays()
    bad = []

    def work(i):
        for k in range(4):
            s = S if (i + k) % 2 else _native.Structures(wl.structures)
            a = _native.query(T, s, P).arrays()
            if any(not np.array_equal(a[c], want[c]) for c in want):
                bad.append((i, k))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert want["count"] > 0 and not bad


@pytest.mark.parametrize("atoms", [1, 511, 512, 513, 1025])
def test_structures_around_a_rank_tile(atoms):
    """Structures cut to sizes around the tiles the axis ranks are sorted in
    (half of them on a coarse grid: equal coordinates across tiles)."""
    from pyjess_gb300 import workloads as W

    structs = _structures(37, [160, 160])
    specs = _templates(37, structs, 20, hi=4)
    for i, s in enumerate(structs):
        for k in ("xyz", "name", "resname", "res_seq", "chain", "serial"):
            s[k] = np.ascontiguousarray(s[k][:atoms])
        if i:
            s["xyz"] = np.round(s["xyz"] / 0.25) * 0.25
    compare(W.pack_templates(specs), W.pack(structs), **PARAMS)


@pytest.mark.parametrize("atoms", [2047, 2048, 2049, 4097])
def test_structures_of_several_rank_tiles(atoms):
    """As test_structures_around_a_rank_tile around multiples of the 2,048
    atoms of a tile, 20 structures at a time (names met by several host
    threads)."""
    from pyjess_gb300 import workloads as W

    structs = _structures(54, [atoms // 6] * 2 + [40] * 18)
    specs = _templates(54, structs, 20, hi=4)
    for i, s in enumerate(structs[:2]):
        for k in ("xyz", "name", "resname", "res_seq", "chain", "serial"):
            s[k] = np.ascontiguousarray(s[k][:atoms])
        assert len(s["xyz"]) == atoms
        if i:
            s["xyz"] = np.round(s["xyz"] / 0.25) * 0.25
    compare(W.pack_templates(specs), W.pack(structs), **PARAMS)


def test_long_lists_replayed():
    """Backbone lists of 4,300 entries with ties (the exact replay in 192 KB of
    shared memory)."""
    from pyjess_gb300 import workloads as W

    structs = _structures(35, [4300])
    for s in structs:
        s["xyz"] = np.round(s["xyz"] / 0.02) * 0.02
    specs = _templates(35, structs, 2, lo=2, hi=3, permissive=True)
    res, ref = compare(W.pack_templates(specs), W.pack(structs), rmsd_threshold=2.0, distance_cutoff=1.0,
                       max_dynamic_distance=1.0)
    assert ref["hits"]["count"] > 0 and res.stats()["leaf_exact"] > 0


def _cut(spec, atoms):
    for k in ("xyz", "res_seq", "chain", "weight", "code", "resnames", "names"):
        setattr(spec, k, getattr(spec, k)[:atoms])
    return spec


@pytest.mark.parametrize("atoms", [32, 33, 63, 64, 65])
@pytest.mark.parametrize("kw", [dict(), dict(mode="fp64"), dict(ignore_chain=2), dict(max_candidates=1),
                                dict(best_match=True, max_candidates=4), dict(reorder=False)])
def test_levels_of_two_lanes(atoms, kw):
    """Templates around 32 and 64 atoms (one level a lane, two, more than
    that), with lists on both sides of the first frontier's room, beside
    ordinary ones."""
    from pyjess_gb300 import workloads as W

    structs = _structures(38, [150, 300])
    specs = [_cut(s, atoms) for s in _templates(38, structs, 4, lo=22, hi=23, radius=16.0)]
    specs += [_cut(s, atoms) for s in _templates(38, structs, 2, lo=17, hi=18, radius=16.0, permissive=True,
                                                 atoms_per_res=4)]
    specs += _templates(40, structs, 6)
    pt = W.pack_templates(specs)
    assert (np.diff(pt.atom_offset) == atoms).sum() >= 2
    _, ref = compare(pt, W.pack(structs), rmsd_threshold=2.0, distance_cutoff=1.6, max_dynamic_distance=1.6, **kw)
    assert (np.diff(ref["hits"]["atom_offset"]) > 32).any() or atoms == 32


@pytest.mark.parametrize("kw", [dict(), dict(max_candidates=20), dict(best_match=True, max_candidates=1000)])
def test_spilled_entries_of_two_lane_levels(kw):
    """As test_spilled_entries with templates of 36 atoms."""
    from pyjess_gb300 import workloads as W

    rng = np.random.default_rng(7)
    structs = W.make_structures([rng], [60], [1])
    specs = [W.make_template(rng, structs[0], 9, modes=(3,), mode_p=(1.0,), radius=14.0, atoms_per_res=4)
             for _ in range(2)]
    compare(W.pack_templates(specs), W.pack(structs), rmsd_threshold=2.0, distance_cutoff=2.0,
            max_dynamic_distance=2.0, **kw)


def _one_seed_any_pair(seed, atoms):
    """One structure and a template of four atoms: the first two have one
    candidate, the others any atom at any distance, so the pair has one item
    and nearly atoms^2 rows."""
    from pyjess_gb300 import workloads as W

    s = _structures(seed, [atoms // 4])[0]
    spec = _templates(seed, [s], 1, lo=4, hi=5, radius=60.0, permissive=True, atoms_per_res=1)[0]
    for k in ("xyz", "name", "resname", "res_seq", "chain", "serial"):
        s[k] = np.array(s[k][:atoms])
    names = sorted({bytes(x) for x in s["name"]})
    s["name"][0], s["name"][20] = np.frombuffer(b"_ZZ__YY_", np.uint8).reshape(2, 4)
    s["chain"][:] = s["chain"][0]
    spec.chain, spec.res_seq = [bytes(s["chain"][0])] * 4, [1, 2, 3, 4]
    spec.names = [[b"_ZZ_"], [b"_YY_"], names, names]
    return W.pack_templates([spec]), W.pack([s])


@pytest.mark.parametrize("atoms", [36, 84, 85, 112])
def test_classes_around_the_largest_counted(atoms):
    """Units whose rows all part at one level, of 370 to 8,302 rows: on
    both sides of the largest class that is counted row by row."""
    pt, ps = _one_seed_any_pair(46, atoms)
    _, ref = compare(pt, ps, rmsd_threshold=100.0, distance_cutoff=300.0, max_dynamic_distance=300.0)
    rows = ref["stats"]["complete"]
    assert ref["hits"]["count"] > 256 and (rows > 4096) == (atoms > 84)


def test_unit_of_half_a_million_rows():
    """One class of hundreds of thousands of rows: ordered within a second
    (each row against every other would take ten)."""
    import time

    pt, ps = _one_seed_any_pair(47, 780)
    kw = dict(rmsd_threshold=7.0, distance_cutoff=300.0, max_dynamic_distance=300.0)
    res, ref = compare(pt, ps, **kw)
    assert ref["hits"]["count"] > 100 and ref["stats"]["complete"] > 500000
    t0 = time.perf_counter()
    gpu_query(pt, ps, **kw)
    assert time.perf_counter() - t0 < 2.0


@pytest.mark.parametrize("kw", [dict(max_candidates=0), dict(max_candidates=40), dict(max_candidates=700),
                                dict(best_match=True, max_candidates=40), dict(best_match=True, max_candidates=700)])
def test_cut_streams_count_the_same_every_time(kw):
    """Items past a pair's cut may or may not have been in flight when its
    earlier ones ended the stream: the counters are of the items before it."""
    from pyjess_gb300 import _native, workloads as W
    from pyjess_gb300._abi import QueryParams

    structs = _structures(45, [1500, 1300, 1400, 1200])
    specs = _templates(45, structs, 12, lo=2, hi=4, permissive=True)
    T, S = _native.Templates(W.pack_templates(specs)), _native.Structures(W.pack(structs))
    P = QueryParams(rmsd_threshold=1.0, distance_cutoff=1.2, max_dynamic_distance=1.2, ignore_chain=0,
                    max_candidates=kw["max_candidates"], best_match=int(kw.get("best_match", False)), reorder=1,
                    mode=_native.MODE_BATCHED_FP32)
    counters = {tuple(_native.query(T, S, P).stats()[k] for k in (
        "partials", "complete", "passing", "hits", "bytes_expansion", "fp64_rechecks")) for _ in range(12)}
    assert len(counters) == 1


@pytest.mark.parametrize("budget", ["1", "60"])
@pytest.mark.parametrize("kw", [dict(), dict(max_candidates=5), dict(best_match=True, max_candidates=7)])
def test_more_items_than_room(monkeypatch, budget, kw):
    """Chunks with more items than there is room for are redone on fewer
    structures, a single structure in order: nothing is refused."""
    from pyjess_gb300 import workloads as W

    monkeypatch.setenv("PJG_ITEM_BUDGET", budget)
    structs = _structures(48, [900, 60, 1500, 700, 800])
    specs = _templates(48, structs, 24, hi=5)
    specs += [_cut(t, 34) for t in _templates(48, structs, 2, lo=12, hi=13, radius=16.0)]
    res, ref = compare(W.pack_templates(specs), W.pack(structs), rmsd_threshold=1.6, distance_cutoff=2.2,
                       max_dynamic_distance=2.2, **kw)
    st = res.stats()
    assert ref["hits"]["count"] > 0 and st["row_splits"] > 0 and st["chunks"] > 1


@pytest.mark.parametrize("structures_a_chunk", [1, 3])
def test_kind_masks_of_a_chunk(monkeypatch, structures_a_chunk):
    """A set with a structure of a thousand atom kinds, whose kind masks do
    not fit a small limit: the masks chunk by chunk."""
    from pyjess_gb300 import workloads as W

    structs = _structures(49, [200, 90, 150, 300, 120, 60, 110])
    s, m = structs[2], 800
    rng = np.random.default_rng(49)
    extra = {"xyz": s["xyz"][rng.integers(len(s["xyz"]), size=m)] + rng.normal(scale=3.0, size=(m, 3)),
             "name": np.frombuffer(b"".join(b"X%03d" % i for i in range(m)), np.uint8).reshape(m, 4),
             "resname": np.tile(np.frombuffer(b"LIG\0", np.uint8), (m, 1)),
             "res_seq": np.arange(900, 900 + m, dtype=np.int32), "chain": np.tile(s["chain"][:1], (m, 1)),
             "serial": np.arange(9000, 9000 + m, dtype=np.int32)}
    for k, v in extra.items():
        s[k] = np.ascontiguousarray(np.concatenate([s[k], v]))
    pt, ps = W.pack_templates(_templates(49, structs, 40)), W.pack(structs)
    kinds = len(np.unique(np.concatenate([s["resname"], s["name"]], 1), axis=0))
    lists = len({(int(c), pt.names[a:b].tobytes(), pt.resnames[e:f].tobytes())
                 for c, a, b, e, f in zip(pt.code, pt.name_offset, pt.name_offset[1:], pt.resname_offset,
                                          pt.resname_offset[1:])})
    monkeypatch.setenv("PJG_MASK_BUDGET", str(structures_a_chunk * lists * 4 * -(-kinds // 32)))
    res, ref = compare(pt, ps, **PARAMS)
    assert ref["hits"]["count"] > 0 and res.stats()["chunks"] == -(-len(structs) // structures_a_chunk)


@pytest.mark.parametrize("atoms", [5, 33])
@pytest.mark.parametrize("max_candidates", [0, 3])
def test_entry_that_cannot_be_split(atoms, max_candidates):
    """Any atom of any residue at any distance: one seed has more children
    than a frontier holds, so the pair goes to the searches in order."""
    from pyjess_gb300 import workloads as W

    structs = _structures(39, [1250])
    names = sorted({bytes(x) for x in structs[0]["name"]})
    spec = _templates(39, structs, 1, lo=atoms, hi=atoms + 1, radius=40.0, permissive=True, atoms_per_res=1)[0]
    spec.names = [list(names) for _ in spec.names]
    assert len(spec.code) == atoms
    _, ref = compare(W.pack_templates([spec]), W.pack(structs), rmsd_threshold=1e3, distance_cutoff=200.0,
                     max_dynamic_distance=200.0, max_candidates=max_candidates, best_match=True)
    assert ref["hits"]["count"] == 1


def test_cut_items_give_the_same_stream_every_time():
    """Hundreds of items of a pair in flight, each asking the ones before it
    whether it is still wanted: the oracle's cut stream in every run."""
    from pyjess_gb300 import workloads as W

    structs = _structures(45, [1500, 1300])
    specs = _templates(45, structs, 6, lo=2, hi=4, permissive=True)
    pt, ps = W.pack_templates(specs), W.pack(structs)
    kw = dict(rmsd_threshold=1.0, distance_cutoff=1.2, max_dynamic_distance=1.2, max_candidates=40)
    _, ref = compare(pt, ps, **kw)
    want = hit_keys(ref["hits"])
    assert len(want) > 0
    for _ in range(20):
        assert hit_keys(gpu_query(pt, ps, **kw).arrays()) == want


@pytest.mark.parametrize("mode", ["fp32", "fp64"])
def test_pair_handed_over_after_rows_of_it_were_written(mode):
    """Twelve ligands, ten of them alone among 30 atoms and the last two in a
    cluster of 8,500: the first item of the pair writes its rows, the second
    meets entries with more children than a frontier holds, and the pair goes
    to the search in order.  Rows and counters are those of one search."""
    from pyjess_gb300 import workloads as W

    rng = np.random.default_rng(53)
    ball = lambda n: (lambda v: v / np.linalg.norm(v, axis=1)[:, None] * rng.uniform(2, 28, (n, 1)))(
        rng.normal(size=(n, 3)))
    centres = np.zeros((12, 3))
    centres[:10, 0] = 1000.0 * np.arange(1, 11)
    centres[10:] = [[0.4, 0.0, 0.0], [-0.4, 0.3, 0.1]]
    ligand = np.array([[0.0, 0.0, 0.0], [1.5, 0.0, 0.2], [0.1, 1.4, 0.3]])
    xyz = np.concatenate([(centres[:, None] + ligand).reshape(-1, 3)] + [centres[i] + ball(30) for i in range(10)] +
                         [ball(8500)])
    n = len(xyz)
    raw = lambda parts, width: np.frombuffer(b"".join(parts), np.uint8).reshape(-1, width).copy()
    s = {"xyz": np.round(xyz, 3), "name": raw([b"_ZZ__YY__XX_"] * 12 + [b"_CA_"] * (n - 36), 4),
         "resname": raw([b"LIG\0"] * 36 + [b"ALA\0"] * (n - 36), 4), "chain": raw([b" A"] * n, 2),
         "res_seq": np.concatenate([np.repeat(np.arange(1, 13), 3), np.arange(100, 100 + n - 36)]).astype(np.int32),
         "serial": np.arange(1, n + 1, dtype=np.int32)}
    spec = W.TemplateSpec(code=[0] * 4, res_seq=[1, 1, 1, 2], chain=[b" A"] * 4,
                          xyz=[*ligand, np.array([9.0, 8.0, 7.0])], weight=[0.0] * 4,
                          names=[[b"_ZZ_"], [b"_YY_"], [b"_XX_"], [b"_CA_"]],
                          resnames=[[b"LIG\0"]] * 3 + [[b"ALA\0"]])
    res, ref = compare(W.pack_templates([spec]), W.pack([s]), mode=mode, rmsd_threshold=5.0, distance_cutoff=20.0,
                       max_dynamic_distance=20.0)
    st = res.stats()
    assert ref["stats"]["complete"] > 17000 and 0 < ref["hits"]["count"] < ref["stats"]["complete"]
    assert st["search_rounds"] == 2 and st["suspensions"] == 1


@pytest.mark.parametrize("max_candidates", [0, 1, 4, 30, 31, 32, 33, 63, 200])
@pytest.mark.parametrize("threshold", [0.75, 1.2])
def test_streams_cut_within_a_step(max_candidates, threshold):
    """Streams of hundreds of rows of which some pass, cut after gaps around
    the 32 rows a warp takes a step."""
    from pyjess_gb300 import workloads as W

    structs = _structures(41, [120, 70])
    specs = _templates(41, structs, 12, lo=2, hi=4, permissive=True)
    _, ref = compare(W.pack_templates(specs), W.pack(structs), rmsd_threshold=threshold, distance_cutoff=2.5,
                     max_dynamic_distance=2.5, max_candidates=max_candidates)
    assert ref["hits"]["count"] > 0


@pytest.mark.parametrize("reach", [1.2, 1.6, 1.9, 2.2])
def test_units_of_dozens_of_rows(reach):
    """Pairs of 2 to 300 rows (every row a hit) in lists of up to 120 entries:
    units on both sides of the rows that each instance holds."""
    from pyjess_gb300 import workloads as W

    structs = _structures(42, [60, 80, 100, 120], chains=1)
    specs = _templates(42, structs, 100, lo=2, hi=4, permissive=True)
    _, ref = compare(W.pack_templates(specs), W.pack(structs), rmsd_threshold=10.0, distance_cutoff=reach,
                     max_dynamic_distance=reach)
    h = ref["hits"]
    rows = np.unique(h["structure"].astype(np.int64) * len(specs) + h["template"], return_counts=True)[1]
    assert (rows > 1).any() and (reach < 1.6 or (rows > 64).any())
