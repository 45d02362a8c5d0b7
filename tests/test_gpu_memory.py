"""Device memory of handles and results: given back when they are dropped."""

import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEPT = 320 << 20  # what the library keeps for its next handles and results, and rounding


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
