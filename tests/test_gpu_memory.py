"""Device memory of handles and results: given back when they are dropped."""

import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEPT = 320 << 20  # what the library keeps for its next handles and results, and rounding


def _in_fresh_threads(n, work):
    """work(i) in n threads one after the other, none of which has used CUDA."""
    import threading

    bad = []

    def run(i):
        try:
            work(i)
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    for i in range(n):
        t = threading.Thread(target=run, args=(i,))
        t.start()
        t.join()
    assert not bad, bad[0]


def test_queries_of_fresh_threads_leave_nothing_behind():
    """A query from each of 80 threads that have never used CUDA: they take
    over what the query before them kept (a stream, a pinned buffer, tens of
    megabytes of blocks), whichever thread that was."""
    import torch

    from pyjess_gb300 import _native, workloads as W
    from pyjess_gb300._abi import QueryParams

    wl = W.config(3, n_structures=60, n_templates=600)
    T, S = _native.Templates(wl.templates), _native.Structures(wl.structures)
    P = QueryParams(rmsd_threshold=2.0, distance_cutoff=1.5, max_dynamic_distance=1.5, max_candidates=-1,
                    ignore_chain=0, best_match=0, reorder=1, mode=_native.MODE_BATCHED_FP32)
    want = _native.query(T, S, P).stats()["hits"]
    hits = []
    one = lambda i: hits.append(_native.query(T, S, P).stats()["hits"])
    _in_fresh_threads(4, one)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _in_fresh_threads(80, one)
    torch.cuda.synchronize()
    assert hits == [want] * 84
    assert free - torch.cuda.mem_get_info()[0] < 128 << 20


def test_handle_dropped_by_a_fresh_thread():
    """The last reference to a handle of 0.8 GB goes in a thread that has
    never used CUDA: its memory is given back all the same."""
    import torch

    from pyjess_gb300 import _native

    _, many = _tiled(3000)
    keep = _native.Structures(_tiled(1)[0])  # (the library's idle streams stay)
    handles = [_native.Structures(many)]
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(6):
        _in_fresh_threads(1, lambda i: handles.pop())
        handles.append(_native.Structures(many))
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 1 << 30
    del keep


def _tiled(copies):
    """One protein `copies` times over."""
    from pyjess_gb300 import workloads as W

    one = W.pack(W.make_structures([np.random.default_rng(51)], [300], [2]))
    n = int(one.atom_offset[-1])
    tile = lambda a: np.tile(a, (copies,) + (1,) * (a.ndim - 1))
    return one, type(one)(atom_offset=np.arange(copies + 1, dtype=np.int64) * n, xyz=tile(one.xyz),
                          name=tile(one.name), resname=tile(one.resname), chain=tile(one.chain),
                          res_seq=tile(one.res_seq), serial=tile(one.serial))


def test_dropped_handles_and_results_leave_the_device(monkeypatch):
    """A result and a structure handle of about a gigabyte each: once
    dropped, other programs of the device can have their memory (the queries'
    own buffers are kept)."""
    import torch

    from pyjess_gb300 import _native, workloads as W
    from pyjess_gb300._abi import QueryParams

    monkeypatch.setenv("PJG_OBJECT_KEEP", str(256 << 20))
    one, many = _tiled(3000)
    rng = np.random.default_rng(52)
    donor = W.make_structures([np.random.default_rng(51)], [300], [2])[0]
    specs = [W.make_template(rng, donor, 3, permissive=True, atoms_per_res=2) for _ in range(2)]
    T = _native.Templates(W.pack_templates(specs))
    P = QueryParams(rmsd_threshold=3.0, distance_cutoff=2.0, max_dynamic_distance=2.0, max_candidates=-1,
                    ignore_chain=0, best_match=0, reorder=1, mode=_native.MODE_BATCHED_FP32)
    want = _native.query(T, _native.Structures(one), P).arrays()
    free = lambda: (gc.collect(), torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[2]
    S = _native.Structures(many)
    res = _native.query(T, S, P)
    hits = res.stats()["hits"]
    assert hits == 3000 * want["count"]
    result_bytes = hits * 152 + 4 * 3000 * len(want["atoms"])
    handle_bytes = 120 * int(many.atom_offset[-1])
    assert min(result_bytes, handle_bytes) > 2 * KEPT
    at = free()
    del res
    after = free()
    assert after - at > result_bytes - KEPT
    del S
    assert free() - after > handle_bytes - KEPT
    again = _native.query(T, _native.Structures(one), P).arrays()
    assert all(np.array_equal(again[k], want[k]) for k in want)
