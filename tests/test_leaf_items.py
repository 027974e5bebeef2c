"""The work items of the leaf pass, built on the host: every source of a round
belongs to one item, and a range is cut by what it costs a lane.

A round of one target computes a second one in vain (a lane carries two), so
its ranges cost as much as those of two targets and are cut as finely.
"""
import ctypes

import numpy as np
import pytest

LEAST, SMS = 128, 148


def _items(harness, tcnt, scnt, near, nmid=0, nsurf=152):
    tcnt, scnt = np.asarray(tcnt, np.int32), np.asarray(scnt, np.int32)
    nptr = np.concatenate([[0], np.cumsum([len(x) for x in near])]).astype(np.int64)
    nidx = np.concatenate(near).astype(np.int32)
    mptr = (np.arange(len(tcnt) + 1) * nmid).astype(np.int64)
    rows = np.zeros((100000, 8), np.int32)
    ns, npart = ctypes.c_int(), ctypes.c_int()
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    n = harness.harness_leaf_items(len(tcnt), p(tcnt), p(scnt), p(nptr), p(nidx), p(mptr), nsurf, LEAST, SMS, p(rows),
                                   len(rows), ctypes.byref(ns), ctypes.byref(npart))
    assert n <= len(rows)
    return rows[:n], nidx, ns.value, npart.value


@pytest.mark.parametrize("nt", [1, 2, 3, 16, 32, 33, 70])
def test_items_cover_every_source_once(harness, nt):
    rng = np.random.default_rng(nt)
    leaves = 40
    scnt = rng.integers(0, 700, leaves)
    near = [rng.integers(0, leaves, 27) for _ in range(leaves)]
    rows, nidx, nsplit, nparts = _items(harness, [nt] * leaves, scnt, near, nmid=3)
    for g in range(leaves):
        for tb in range(0, nt, 32):
            it = rows[(rows[:, 0] == g) & (rows[:, 1] == tb)]
            got = []
            for _, _, nb, nn, skip, take, _, _ in it:
                src = np.concatenate([np.arange(scnt[s]) + 1000 * (nb + k) for k, s in enumerate(nidx[nb:nb + nn])] or [[]])
                assert take <= len(src) - (skip if nn else 0)
                got.append(src[skip:skip + take])
            want = np.concatenate([np.arange(scnt[s]) + 1000 * (27 * g + k) for k, s in enumerate(near[g])])
            assert np.array_equal(np.concatenate(got), want)
            assert it[:, 6].sum() == 3
    assert sorted(rows[rows[:, 7] >= 0][:, 7]) == list(range(nparts))


def test_a_round_of_one_target_is_cut_like_one_of_two(harness):
    scnt = [4000] * 60
    near = [np.arange(60)] * 60
    count = [len(_items(harness, [nt] * 60, scnt, near)[0]) for nt in (1, 2)]
    mixed, *_ = _items(harness, [1, 2] * 30, scnt, near)
    one, two = (np.sum(mixed[:, 0] % 2 == k) for k in (0, 1))
    assert count[0] == count[1] and one == two
