"""pjg_superpose_noalloc: the allocation-free superposition entry point.

Callers that cannot allocate device memory while they run (a real-time
loop, an application whose memory manager owns every device allocation) pass
their own input and output buffers; the entry point's only scratch is a
static device array inside the library.  This test
calls it through the C ABI on the hits of a normal `pjg_query` and checks that
it reproduces that query's rmsd, rotations and centroids, twice in a row
(the second call reuses the static scratch left by the first).  The file is
named so that pytest collects it last.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RMSD_TOL = 1e-9
ROT_TOL = 1e-7


def _bind():
    from pyjess_gb300 import _native

    L = _native.init()
    f = L.pjg_superpose_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_int32, C.c_double, C.c_void_p, C.c_void_p,
                  C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
    L.pjg_noalloc_last_error.restype = C.c_char_p
    return L


def test_superpose_noalloc_matches_query(golden):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from pyjess_gb300 import Jess, Molecule, Template, _native
    from pyjess_gb300._abi import QueryParams
    from pyjess_gb300._pack import pack_molecules

    L = _bind()
    amy = Molecule.load(str(golden / "1AMY.pdb"))
    t133 = Template.load(str(golden / "1.3.3.tpl"))
    t412 = Template.load(str(golden / "4.1.2.tpl"))
    jess = Jess([t133, t412])
    pt = jess._packed_templates()
    ps = pack_molecules([amy])
    P = QueryParams(rmsd_threshold=2.0, distance_cutoff=4.0, max_dynamic_distance=4.0, max_candidates=-1,
                    ignore_chain=0, best_match=0, reorder=1, mode=_native.MODE_BATCHED_FP32)
    ref = _native.query(_native.Templates(pt), _native.Structures(ps), P).arrays()
    assert ref["count"] > 100

    dev = torch.device("cuda")
    for t in range(pt.n_templates):
        rows = np.flatnonzero(ref["template"] == t)
        if len(rows) == 0:
            continue
        n = int(pt.atom_offset[t + 1] - pt.atom_offset[t])
        atoms = np.stack([ref["atoms"][ref["atom_offset"][i]:ref["atom_offset"][i + 1]] for i in rows])
        mol = torch.tensor(ps.xyz[atoms].reshape(-1), dtype=torch.float64, device=dev)
        tpl = torch.tensor(pt.xyz[pt.atom_offset[t]:pt.atom_offset[t + 1]].reshape(-1), dtype=torch.float64,
                           device=dev)
        m = len(rows)
        rmsd = torch.empty(m, dtype=torch.float64, device=dev)
        rot = torch.empty(9 * m, dtype=torch.float64, device=dev)
        cen = torch.empty(6 * m, dtype=torch.float64, device=dev)
        pass_rows = torch.empty(m, dtype=torch.int32, device=dev)
        pass_count = torch.empty(1, dtype=torch.int32, device=dev)
        # second call: a threshold between the hits' rmsds, so the ordered
        # compaction keeps a strict subset
        thresholds = (2.0, float(np.median(ref["rmsd"][rows])))
        for threshold in thresholds:
            torch.cuda.synchronize()
            st = L.pjg_superpose_noalloc(mol.data_ptr(), tpl.data_ptr(), m, n, threshold, rmsd.data_ptr(),
                                         rot.data_ptr(), cen.data_ptr(), pass_rows.data_ptr(),
                                         pass_count.data_ptr(), None)
            assert st == 0, L.pjg_noalloc_last_error()
            torch.cuda.synchronize()
            r = rmsd.cpu().numpy()
            assert np.abs(r - ref["rmsd"][rows]).max() <= RMSD_TOL
            assert np.abs(rot.cpu().numpy().reshape(m, 9) - ref["rotation"][rows]).max() <= ROT_TOL
            assert np.abs(cen.cpu().numpy().reshape(m, 6) - ref["centres"][rows]).max() <= 1e-9
            expect = np.flatnonzero(ref["rmsd"][rows] <= threshold)
            k = int(pass_count.cpu().item())
            assert k == len(expect)
            assert np.array_equal(pass_rows.cpu().numpy()[:k], expect)


def test_superpose_noalloc_rejects_oversize():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    L = _bind()
    count = torch.empty(1, dtype=torch.int32, device="cuda")
    st = L.pjg_superpose_noalloc(None, None, (1 << 20) + 1, 9, 2.0, None, None, None, None, count.data_ptr(), None)
    assert st == 1
    assert b"at most" in L.pjg_noalloc_last_error()


@pytest.mark.parametrize("rows, atoms", [(0, 3), (1, 3), (31, 32), (32, 12), (33, 2), (64, 5), (65, 1), (1023, 9),
                                         (1025, 12), (33000, 4)])
def test_superpose_noalloc_row_edges(rows, atoms):
    """Row counts around a warp, a block and the compaction's 1,024-row tiles
    against numpy's SVD fit (FP64, rmsd and rotation within the bounds of the
    query tests), and the rows under the threshold in row order."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    L = _bind()
    rng = np.random.default_rng([77, rows, atoms])
    tpl = rng.normal(scale=4.0, size=(atoms, 3))
    mol = tpl + rng.normal(size=(rows, atoms, 3)) * rng.uniform(0.1, 2.0, size=(rows, 1, 1))
    ca, cb = mol.mean(1), tpl.mean(0)
    u, sv, vt = np.linalg.svd(np.einsum("ni,mnj->mij", tpl - cb, mol - ca[:, None]))
    sign = np.ones((rows, 3))
    sign[:, 2] = np.sign(np.linalg.det(u) * np.linalg.det(vt))
    R = np.einsum("mij,mj,mjk->mik", u, sign, vt)
    want = np.sqrt((((tpl - cb) - np.einsum("mij,mnj->mni", R, mol - ca[:, None])) ** 2).sum((1, 2)) / atoms)
    dev = torch.device("cuda")
    m = max(rows, 1)
    d = [torch.tensor(mol.reshape(-1), device=dev), torch.tensor(tpl.reshape(-1), device=dev)]
    rmsd, rot, cen = (torch.zeros(k * m, dtype=torch.float64, device=dev) for k in (1, 9, 6))
    idx, count = (torch.full((k,), -1, dtype=torch.int32, device=dev) for k in (m, 1))
    thr = float(np.median(want)) + 1e-7 if rows else 1.0
    st = L.pjg_superpose_noalloc(d[0].data_ptr(), d[1].data_ptr(), rows, atoms, thr, rmsd.data_ptr(), rot.data_ptr(),
                                 cen.data_ptr(), idx.data_ptr(), count.data_ptr(), None)
    assert st == 0, L.pjg_noalloc_last_error()
    torch.cuda.synchronize()
    expect = np.flatnonzero(want <= thr) if atoms >= 3 else np.zeros(0, int)  # fewer atoms: no defined rotation
    k = int(count.item())
    assert k == len(expect) and np.array_equal(idx.cpu().numpy()[:k], expect)
    if rows:
        assert np.abs(rmsd.cpu().numpy() - want).max() <= RMSD_TOL if atoms >= 3 else True
        assert np.abs(cen.cpu().numpy().reshape(rows, 6)[:, :3] - ca).max() <= 1e-9
    if rows and atoms >= 4:  # (well separated singular values: a defined rotation)
        ok = (sv[:, 1] + sign[:, 2] * sv[:, 2]) > 1e-3 * sv[:, 0]
        assert np.abs(rot.cpu().numpy().reshape(rows, 3, 3) - R)[ok].max() <= ROT_TOL


@pytest.mark.parametrize("atoms", [5, 12, 17, 31, 32])
def test_superpose_noalloc_centres_are_tree_sums(atoms):
    """One coordinate of 1 among ones of 2^-53, which a running sum loses one
    by one: the centres are within the roundings of a tree of the atoms (five
    additions on the way of any of them, then the division)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    L = _bind()
    u = 2.0 ** -53
    mol = np.full((atoms, atoms, 3), u)  # row r: the 1 at atom r
    mol[np.arange(atoms), np.arange(atoms)] = 1.0
    exact = (1 + (atoms - 1) * 2.0 ** -53) / atoms  # (in units of the last place: the roundings below cover its own)
    dev = torch.device("cuda")
    d = [torch.tensor(mol.reshape(-1), device=dev), torch.tensor(mol[0].reshape(-1), device=dev)]
    rmsd, rot, cen = (torch.zeros(k * atoms, dtype=torch.float64, device=dev) for k in (1, 9, 6))
    idx, count = (torch.zeros(k, dtype=torch.int32, device=dev) for k in (atoms, 1))
    st = L.pjg_superpose_noalloc(d[0].data_ptr(), d[1].data_ptr(), atoms, atoms, 1.0, rmsd.data_ptr(), rot.data_ptr(),
                                 cen.data_ptr(), idx.data_ptr(), count.data_ptr(), None)
    assert st == 0, L.pjg_noalloc_last_error()
    torch.cuda.synchronize()
    err = np.abs(cen.cpu().numpy().reshape(atoms, 6) - exact).max()
    assert err <= (5 * u * (1 + atoms * u) + 2 * u) / atoms, err * atoms / u
