"""Host calls with outputs decoded on the device against the raw fixed-point
calls decoded on the host: the same bits, for results that come back in one
staged copy and for larger ones, every output selection, and after an error."""

import numpy as np
import pytest
import torch

from tests.helpers import f32_round
from timemachine_b200 import _lib
from timemachine_b200 import potentials as P
from timemachine_b200 import testsystems
from timemachine_b200.batch import ReplicaBatch
from timemachine_b200.fixed_point import du_dp_fixed_to_float, fixed_to_float, sum_fixed

pytestmark = pytest.mark.gpu


def _want(impl, x, p, box, lam, flags, columns):
    dx, dp, dl, u = impl._execute_fixed(x, p, box, lam, *flags)
    decode = du_dp_fixed_to_float if columns else fixed_to_float
    return (
        None if dx is None else fixed_to_float(dx),
        None if dp is None else decode(dp).reshape(p.shape),
        None if dl is None else fixed_to_float(sum_fixed(dl)),
        None if u is None else fixed_to_float(sum_fixed(u)),
    )


def _same(got, want):
    for a, b in zip(got, want):
        assert (a is None) == (b is None)
        if a is not None:
            np.testing.assert_array_equal(np.asarray(a), np.asarray(b))


@pytest.mark.parametrize("n", [300, 6100])  # below and above the staged copy's size
@pytest.mark.parametrize("interpolated", [False, True])
def test_potential_calls(n, interpolated):
    s = testsystems.system_of_size(n, seed=n, n_ligand=12, min_edge=2.9)
    x, p = f32_round(s.x), f32_round(s.params)
    cls = P.NonbondedInterpolated if interpolated else P.Nonbonded
    if interpolated:
        p = np.concatenate([p, 1.1 * p])
    impl = cls(s.exclusion_idxs, s.scales, s.lambda_plane_idxs, s.lambda_offset_idxs, s.beta, s.cutoff)
    impl = impl.unbound_impl(np.float32)
    for flags in P.all_flag_combinations():
        _same(impl.execute_selective(x, p, s.box, 0.3, *flags), _want(impl, x, p, s.box, 0.3, flags, True))
    lams = np.linspace(0, 1, 3)
    frames = np.stack([x, f32_round(x + 0.2)])
    boxes = np.stack([s.box, s.box])
    got = impl.execute_selective_batch(frames, np.stack([p, 0.9 * p]), boxes, lams, True, True, True, True)
    for c, pb, k in [(0, 0, 0), (0, 1, 2), (1, 0, 1), (1, 1, 2)]:
        want = _want(impl, frames[c], [p, 0.9 * p][pb], s.box, lams[k], (True,) * 4, True)
        _same([g[c, pb, k] for g in got], want)
    windows = impl.execute_windows(x, p, s.box, lams)
    _same([g[1] for g in windows], _want(impl, x, p, s.box, lams[1], (True,) * 4, True))
    with pytest.raises(RuntimeError, match="Cutoff with padding is more than half"):
        impl.execute(x, p, np.eye(3) * 2.0, 0.3)
    _same(impl.execute(x, p, s.box, 0.3), _want(impl, x, p, s.box, 0.3, (True,) * 4, True))
    with pytest.raises(RuntimeError):
        impl.execute_windows(x, p, s.box, np.linspace(0, 1, 33))
    bonds = P.HarmonicBond(s.bond_idxs).unbound_impl(np.float32)
    _same(bonds.execute(x, s.bond_params, s.box, 0.0), _want(bonds, x, s.bond_params, s.box, 0.0, (True,) * 4, False))


def test_replica_results():
    b = ReplicaBatch()
    systems = [testsystems.system_of_size(n, seed=n, n_ligand=10, min_edge=2.9) for n in (400, 2600, 900)]
    ids = [b.add(s, 0.4) for s in systems]
    b.evaluate()
    for rid, s in zip(ids, systems):
        dx, dp, dl, u = b.result_fixed(rid)
        want = fixed_to_float(dx), du_dp_fixed_to_float(dp), fixed_to_float(sum_fixed(dl)), fixed_to_float(sum_fixed(u))
        _same(b.result(rid), want)


def test_replica_results_after_a_change_of_priority():
    """The workspace of the results outlives the stream it was allocated on: it
    grows and is freed on the batch's current one."""
    b = ReplicaBatch()
    ids = []
    for n, priority in ((300, -1), (2600, 0), (5000, None)):  # each larger: the workspace grows
        s = testsystems.system_of_size(n, seed=n, n_ligand=10, min_edge=2.9)
        ids.append(b.add(s, 0.4))
        b.evaluate()
        for rid in ids:
            dx, dp, dl, u = b.result_fixed(rid)
            want = fixed_to_float(dx), du_dp_fixed_to_float(dp), fixed_to_float(sum_fixed(dl)), fixed_to_float(sum_fixed(u))
            _same(b.result(rid), want)
        if priority is not None:
            _lib.check(b._lib.tmnb_batch_set_priority(b._h, priority))
    del b
    torch.cuda.synchronize()  # raises what the frees may have left
