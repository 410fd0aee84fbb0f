"""The tile walk of the pair kernel, and the list rebuild before it, against the pair-list kernel over the same
pairs: every output is an exact integer sum of per-pair fixed-point values, and
both kernels round a pair the same way, so they agree bit for bit. Sizes sit at
the edges of tiles and row groups; coordinates lie in several periodic images
(one-image shift and general minimum image); random positions bring pairs whose
terms exceed the shared-memory limbs; a dense group fills the list builder's
column buffer."""

import numpy as np
import pytest
import torch
from scipy.spatial import cKDTree

from tests.gpu_helpers import to_dev
from tests.helpers import f32_round, random_params
from timemachine_b200 import potentials as P
from timemachine_b200 import testsystems
from timemachine_b200.fixed_point import fixed_to_float

pytestmark = pytest.mark.gpu


def _case(n, seed, images):
    rng = np.random.default_rng(seed)
    edges = np.array([3.1, 3.4, 5.3])
    x = rng.uniform(0, 1, size=(n, 3)) * edges
    x = x + rng.integers(-images, images + 1, size=(n, 3)) * edges
    params = random_params(rng, n)
    params[rng.random(n) < 0.6, 2] = 0.0  # most atoms without Lennard-Jones terms, as in water
    plane = rng.integers(-1, 2, size=n).astype(np.int32) * (rng.random(n) < 0.1)
    offset = rng.integers(-1, 2, size=n).astype(np.int32) * (rng.random(n) < 0.1)
    return f32_round(x), f32_round(params), np.diag(edges), plane.astype(np.int32), offset.astype(np.int32)


def _fixed(impl, x, p, box, lam, flags=(True, True, True, True)):
    out = impl._execute_fixed(x, p, box, lam, *flags)
    # per-atom energies and du_dl: only their sums are defined
    return [None if o is None else (o if k < 2 else o.sum(dtype=np.uint64)) for k, o in enumerate(out)]


def _assert_same(a, b):
    for name, u, v in zip(("du_dx", "du_dp", "du_dl", "u"), a, b):
        if u is not None:
            np.testing.assert_array_equal(u, v, err_msg=name)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 65, 257, 1001])
@pytest.mark.parametrize("rows,precision", [(8, np.float32), (16, np.float32), (32, np.float32), (16, np.float64)])
@pytest.mark.parametrize("images", [0, 3])
def test_all_pairs_equals_pair_list(n, rows, precision, images):
    x, p, box, plane, offset = _case(n, 100 * n + images, images)
    cutoff, beta = 1.2, 2.0
    impl = P.NonbondedAllPairs(plane, offset, beta, cutoff).unbound_impl(precision)
    if precision == np.float32:
        impl.set_tile_rows(rows)
    i, j = np.triu_indices(n, 1)
    pairs = np.stack([i, j], axis=1).astype(np.int32)
    ref = P.NonbondedPairList(pairs, np.ones((len(pairs), 2)), plane, offset, beta, cutoff).unbound_impl(precision)
    want = _fixed(ref, x, p, box, 0.3)
    _assert_same(_fixed(impl, x, p, box, 0.3), want)
    # moved within the list's padding: the columns keep the order of the old distances
    moved = f32_round(x + np.random.default_rng(n).uniform(-0.02, 0.02, size=x.shape))
    _assert_same(_fixed(impl, moved, p, box, 0.3), _fixed(ref, moved, p, box, 0.3))
    for flags in P.all_flag_combinations():
        if any(flags):
            _assert_same(_fixed(impl, moved, p, box, 0.3, flags), _fixed(ref, moved, p, box, 0.3))


@pytest.mark.parametrize("interpolated", [False, True])
def test_dense_group_fills_the_column_buffer(interpolated):
    """16 + 3 row atoms with about 6,000 column atoms in reach: more than the
    list builder sorts; the others follow unsorted."""
    n, nr = 6019, 19
    rng = np.random.default_rng(5)
    edge = 3.0
    x = rng.uniform(0, edge, size=(n, 3))
    x[:nr] = edge / 2 + rng.uniform(-0.1, 0.1, size=(nr, 3))
    x = f32_round(x)
    params = f32_round(random_params(rng, n))
    if interpolated:
        params = np.concatenate([params, f32_round(params * rng.uniform(0.5, 1.5, size=params.shape))])
    plane = np.zeros(n, np.int32)
    offset = (np.arange(n) < 5).astype(np.int32)
    box, cutoff, beta = np.eye(3) * edge, 1.39, 2.0
    rows = np.arange(nr, dtype=np.int32)
    pairs = np.stack(np.meshgrid(rows, np.arange(nr, n), indexing="ij"), axis=-1).reshape(-1, 2).astype(np.int32)
    group = P.NonbondedInteractionGroupInterpolated if interpolated else P.NonbondedInteractionGroup
    plist = P.NonbondedPairListInterpolated if interpolated else P.NonbondedPairList
    impl = group(rows, plane, offset, beta, cutoff).unbound_impl(np.float32)
    ref = plist(pairs, np.ones((len(pairs), 2)), plane, offset, beta, cutoff).unbound_impl(np.float32)
    for lam in (0.0, 0.4):
        _assert_same(_fixed(impl, x, params, box, lam), _fixed(ref, x, params, box, lam))
    _, tiles, _ = impl.get_nblist()
    got = [np.sort(t) for t in tiles]
    assert max(len(t) for t in got) > 3072
    assert all(len(np.unique(t)) == len(t) for t in got)


@pytest.mark.parametrize("n", [255, 8192, 8193, 32768, 32769, 131105])
def test_rebuild_paths(n):
    """Sizes at the edges of the three ways a call prepares and sorts, and one whose
    column blocks the tile build goes through in two passes (4,096 each): the list
    that each leaves gives the pair list's sums, with and without the Hilbert
    order, after the atoms have moved and with other windows per call."""
    rng = np.random.default_rng(n)
    edge = max(2.0, (n / 100.0) ** (1.0 / 3.0))
    cutoff, beta = 0.4, 2.0
    box = np.eye(3) * edge
    p = f32_round(random_params(rng, n))
    plane, offset = np.zeros(n, np.int32), (rng.random(n) < 0.002).astype(np.int32)
    impl = P.NonbondedAllPairs(plane, offset, beta, cutoff).unbound_impl(np.float32)
    plain = P.NonbondedAllPairs(plane, offset, beta, cutoff).unbound_impl(np.float32)
    plain.disable_hilbert_sort()
    for _ in range(2):
        x = f32_round(rng.uniform(0, edge, size=(n, 3)))
        wrapped = np.minimum(x - edge * np.floor(x / edge), np.nextafter(edge, 0))
        pairs = cKDTree(wrapped, boxsize=edge).query_pairs(cutoff + 1e-3, output_type="ndarray").astype(np.int32)
        ref = P.NonbondedPairList(pairs, np.ones((len(pairs), 2)), plane, offset, beta, cutoff).unbound_impl(np.float32)
        want = _fixed(ref, x, p, box, 0.3)
        _assert_same(_fixed(impl, x, p, box, 0.3), want)
        _assert_same(_fixed(plain, x, p, box, 0.3), want)
    multi = impl.execute_windows_fixed(x, p, box, np.array([0.3, 0.9]))
    _assert_same([multi[k][0] if k < 2 else multi[k][0].sum(dtype=np.uint64) for k in range(4)], want)
    energy = _fixed(impl, x, p, box, 0.3, (False, False, False, True))
    _assert_same(energy, want)


@pytest.mark.parametrize("n", [6000, 33000])  # the sort in one cluster, and as three kernels
def test_only_compact_sites_take_the_first_slots(n):
    """Atoms with a lambda offset sit in the first slots where they lie together;
    where they lie in two places or anywhere, row groups that held several of them
    would list the columns around all (of two places 1.3 times, of many over twice
    the widest list without the rule), so after the first rebuild they keep the
    plain order. The sums are the pair list's either way."""
    s = testsystems.system_of_size(n, seed=n, n_ligand=40)
    x, p, N = f32_round(s.x), f32_round(s.params), s.N
    far = np.argsort((np.minimum(s.x, np.diag(s.box) - s.x) ** 2).sum(axis=1))[:24]  # a corner of the box
    layouts = {
        "none": [],
        "ligand": s.ligand_idxs,
        "two": np.concatenate([s.ligand_idxs, far]),
        "anywhere": np.random.default_rng(n).choice(N, N // 100, replace=False),
    }
    plane, widest = np.zeros(N, np.int32), {}
    for name, idxs in layouts.items():
        offset = np.zeros(N, np.int32)
        offset[idxs] = 1
        impl = P.NonbondedAllPairs(plane, offset, s.beta, s.cutoff).unbound_impl(np.float32)
        plain = P.NonbondedAllPairs(plane, offset, s.beta, s.cutoff).unbound_impl(np.float32)
        plain.disable_hilbert_sort()
        for shift in (0.0, 0.3, 0.0):
            _assert_same(_fixed(impl, f32_round(x + shift), p, s.box, 0.3), _fixed(plain, f32_round(x + shift), p, s.box, 0.3))
        perm, tiles, _ = impl.get_nblist()
        assert np.array_equal(np.sort(perm), np.arange(N))
        widest[name] = max(len(t) for t in tiles)
        together = set(perm[: len(idxs) // 16 * 16]) <= set(idxs)  # full row groups
        assert together == (name in ("none", "ligand"))
    print(widest)
    for name in ("ligand", "two", "anywhere"):
        assert widest[name] <= 1.2 * widest["none"]
    # many windows and many such atoms: first wherever they are
    offset = np.zeros(N, np.int32)
    offset[np.random.default_rng(n).choice(N, N // 30, replace=False)] = 1
    impl = P.NonbondedAllPairs(plane, offset, s.beta, s.cutoff).unbound_impl(np.float32)
    for shift in (0.0, 0.3):
        multi = impl.execute_windows_fixed(f32_round(x + shift), p, s.box, np.array([0.3, 0.9]))
        assert set(impl.get_nblist()[0][: N // 30 // 16 * 16]) <= set(np.flatnonzero(offset))
    plain = P.NonbondedAllPairs(plane, offset, s.beta, s.cutoff).unbound_impl(np.float32)
    plain.disable_hilbert_sort()
    _assert_same([multi[k][0] if k < 2 else multi[k][0].sum(dtype=np.uint64) for k in range(4)],
                 _fixed(plain, f32_round(x + 0.3), p, s.box, 0.3))


@pytest.mark.parametrize("n", [200, 3000, 9000])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_an_atom_without_a_position_pairs_with_none(n, value):
    """One coordinate of an atom is not a number; the others keep all their pairs,
    also those that share its row group and its block. The atom is alone in having
    a lambda offset, so it is the first of its group."""
    s = testsystems.system_of_size(n, seed=n, n_ligand=5, min_edge=2.9)
    x, p, N = f32_round(s.x), f32_round(s.params), s.N
    plane, offset = np.zeros(N, np.int32), np.zeros(N, np.int32)
    lost = int(s.ligand_idxs[2])
    offset[lost] = 1
    rest = np.arange(N) != lost
    ref = P.NonbondedAllPairs(plane[rest], offset[rest], s.beta, s.cutoff).unbound_impl(np.float32)
    want = _fixed(ref, x[rest], p[rest], s.box, 0.0)
    for axis in range(3):
        y = x.copy()
        y[lost, axis] = value
        for precision in (np.float32, np.float64):
            impl = P.NonbondedAllPairs(plane, offset, s.beta, s.cutoff).unbound_impl(precision)
            dx, dp, dl, u = _fixed(impl, y, p, s.box, 0.0)
            assert not dx[lost].any() and not dp.reshape(N, 3)[lost].any()
            if precision == np.float32:
                _assert_same((dx[rest], dp.reshape(N, 3)[rest].reshape(-1), dl, u), want)
            else:
                np.testing.assert_allclose(fixed_to_float(u), fixed_to_float(want[3]), rtol=1e-5)


@pytest.mark.parametrize("interpolated", [False, True])
def test_pair_list_outputs_do_not_carry_over(interpolated):
    """A pair list clears the accumulators of the outputs it was asked for; calls
    with other outputs and windows in between find all of them at zero."""
    x, p, box, plane, offset = _case(300, 1, 0)
    if interpolated:
        p = np.concatenate([p, f32_round(1.2 * p)])
    rng = np.random.default_rng(3)
    pairs = np.array([c for c in rng.integers(0, 300, size=(900, 2)) if c[0] != c[1]], dtype=np.int32)
    cls = P.NonbondedPairListInterpolated if interpolated else P.NonbondedPairList
    make = lambda: cls(pairs, np.ones((len(pairs), 2)), plane, offset, 2.0, 1.2).unbound_impl(np.float32)
    want = _fixed(make(), x, p, box, 0.3)
    impl = make()
    flags = [f for f in P.all_flag_combinations() if any(f)]
    for k in rng.permutation(np.repeat(np.arange(len(flags)), 3)):
        _assert_same(_fixed(impl, x, p, box, 0.3, flags[k]), [w if f else None for w, f in zip(want, flags[k])])
        if k % 4 == 0:
            multi = impl.execute_windows_fixed(x, p, box, np.array([0.3, 0.9]))
            _assert_same([multi[j][0] if j < 2 else multi[j][0].sum(dtype=np.uint64) for j in range(4)], want)


def test_long_items_flush_between_tiles_left_out():
    """32 rows and four tiles per item (several windows, from 40,000 atoms on): the row
    sums are flushed in the middle of an item, whose lambda-dependent tiles are left
    out and evaluated per window. Equal to 16 rows, one window at a time."""
    s = testsystems.system_of_size(40500, seed=11, n_ligand=40)
    x, p = f32_round(s.x), f32_round(s.params)
    offset = s.lambda_offset_idxs.copy()
    offset[np.random.default_rng(4).choice(s.N, 30, replace=False)] = 1  # lambda-dependent tiles in many items
    lams = np.array([0.2, 0.7])
    impl = P.NonbondedAllPairs(s.lambda_plane_idxs, offset, s.beta, s.cutoff).unbound_impl(np.float32)
    one = P.NonbondedAllPairs(s.lambda_plane_idxs, offset, s.beta, s.cutoff).unbound_impl(np.float32)
    impl.set_tile_rows(32)
    got = impl.execute_windows_fixed(x, p, s.box, lams)
    tiles, items, _ = impl.nblist_stats()
    assert tiles > 3 * items  # most items hold four
    for k, lam in enumerate(lams):
        want = _fixed(one, x, p, s.box, lam)
        _assert_same([got[j][k] if j < 2 else got[j][k].sum(dtype=np.uint64) for j in range(4)], want)


def test_the_first_slots_are_tried_again():
    """After a wide row group 1,000 rebuilds keep the plain order, then the atoms take
    the first slots once more."""
    s = testsystems.system_of_size(3000, seed=2, n_ligand=20)
    offset = np.zeros(s.N, np.int32)
    offset[np.random.default_rng(1).choice(s.N, 64, replace=False)] = 1
    impl = P.NonbondedAllPairs(np.zeros(s.N, np.int32), offset, s.beta, s.cutoff).unbound_impl(np.float32)
    frames = [to_dev(s.x), to_dev(s.x + 0.3)]
    p, box = to_dev(s.params).reshape(-1), to_dev(s.box)
    out = torch.zeros((s.N, 3), dtype=torch.int64, device="cuda")
    first = []
    for k in range(1004):
        impl.execute_device(frames[k % 2], p, box, 0.3, out)
        if k in (0, 1, 2, 500, 999, 1000, 1001, 1002, 1003):
            torch.cuda.synchronize()
            perm, _, _ = impl.get_nblist()
            if set(perm[:64]) == set(np.flatnonzero(offset)):
                first.append(k)
    assert impl.nblist_stats()[2] == 1004  # every call rebuilt
    assert first == [0, 1001]


def test_rebuild_of_wide_lists_costs_one_pass():
    """At 1.6 nm many row groups list more columns than the builder sorts. A
    rebuilding energy call of 5,000 atoms took twice one that keeps its list before
    the columns were sorted, 2.9 times when such a group was done again in rounds, and
    takes 2.2 times now."""
    n, edge, cutoff = 5000, 50.0 ** (1.0 / 3.0), 1.6
    rng = np.random.default_rng(0)
    g = (np.arange(18) + 0.5) * edge / 18
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    x = x[rng.choice(len(x), n, replace=False)] + rng.normal(scale=0.02, size=(n, 3))
    p = np.stack([rng.normal(size=n), np.full(n, 0.15), np.where(np.arange(n) % 3 == 0, 0.8, 0.0)], axis=1)
    zero = np.zeros(n, np.int32)
    impl = P.NonbondedAllPairs(zero, zero, 2.0, cutoff).unbound_impl(np.float32)
    frames = [to_dev(x), to_dev(x + 0.3)]
    dp, box, u = to_dev(p).reshape(-1), to_dev(np.eye(3) * edge), torch.zeros(n, dtype=torch.int64, device="cuda")

    def us(moving):
        best = np.inf
        for _ in range(6):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            for k in range(20):
                impl.execute_device(frames[k % 2 if moving else 0], dp, box, 0.3, None, None, None, u)
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end) / 20 * 1e3)
        return best

    kept, rebuilt = us(False), us(True)
    assert max(len(t) for t in impl.get_nblist()[1]) > 3072
    print(f"list kept {kept:.1f} us, rebuilt {rebuilt:.1f} us")
    assert rebuilt < 2.7 * kept
