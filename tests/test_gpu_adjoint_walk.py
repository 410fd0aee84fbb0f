"""The adjoint kernel's tile walk at the edges of tiles and row groups and over
periodic images, against the FP64 double-backward oracle; and the upstream
gradient of du_dl given as a float and as a device value."""

import numpy as np
import pytest
import torch

from oracle.nonbonded_oracle import force_vjp_oracle
from tests.gpu_helpers import to_dev
from tests.helpers import f32_round, small_water_case
from timemachine_b200 import potentials as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 15, 16, 17, 33, 95, 600])
@pytest.mark.parametrize("rows", [8, 16, 32])
def test_walk_against_oracle(n, rows):
    rng = np.random.default_rng(n)
    c = small_water_case(rng, n, planes=(-1, 2), offsets=(-1, 2))
    few = rng.random(n) < 0.2  # most tiles hold no lambda-dependent atom
    plane, offset = (np.where(few, c[k], 0).astype(np.int32) for k in ("plane", "offset"))
    x = f32_round(c["x"] + rng.integers(-2, 3, size=(n, 3)) * np.diag(c["box"]))
    p = f32_round(c["params"])
    p[rng.random(n) < 0.5, 2] = 0.0
    G, g, lam, beta, cutoff = rng.normal(size=(n, 3)), 0.7, 0.4, 2.0, 1.2
    excl, scales = c["exclusion_idxs"], c["scales"]
    impl = P.Nonbonded(excl, scales, plane, offset, beta, cutoff).unbound_impl(np.float32)
    impl.set_tile_rows(rows)
    got = []
    for upstream in (g, torch.tensor(g, dtype=torch.float64, device="cuda")):
        gp = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
        gw = torch.zeros(n, dtype=torch.float64, device="cuda")
        impl.adjoint_device(to_dev(x), to_dev(p).reshape(-1), to_dev(c["box"]), lam, to_dev(G), upstream, gp, gw)
        got.append((gp.cpu().numpy().reshape(n, 3), gw.cpu().numpy()))
    _, rp, rw = force_vjp_oracle(x, p, c["box"], lam, plane, offset, beta, cutoff, excl, scales, G, g)
    # the kernel leaves sig / eps of pairs without both epsilons at zero, as the
    # oracle does; FP64 on both sides: n terms of ~1e-16 relative error each
    for gp, gw in got:
        for ref, val in ((rp, gp), (rw, gw)):
            assert np.max(np.abs(ref - val)) <= 1e-10 * max(1.0, np.max(np.abs(ref)))


def test_upstream_value_still_being_computed_while_another_stream_is_named():
    """The upstream gradient of du_dl is taken in the order of the stream that
    computes it, and its memory may go to another tensor after the call."""
    n = 600
    c = small_water_case(np.random.default_rng(n), n, planes=(-1, 2), offsets=(-1, 2))
    impl = P.Nonbonded(c["exclusion_idxs"], c["scales"], c["plane"], c["offset"], 2.0, 1.2).unbound_impl(np.float32)
    x, p, box = to_dev(f32_round(c["x"])), to_dev(f32_round(c["params"])).reshape(-1), to_dev(c["box"])
    G = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    side = torch.cuda.Stream()

    def vjp(g, **kw):
        gp, gw = torch.zeros(3 * n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        g = g()
        impl.adjoint_device(x, p, box, 0.4, G, g, gp, gw, **kw)
        del g
        torch.full((1,), 5.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return gp.cpu().numpy(), gw.cpu().numpy()

    def late():  # 0.7, some milliseconds from now
        g = torch.zeros(1, dtype=torch.float64, device="cuda")
        torch.cuda._sleep(20_000_000)
        return g.add_(0.7)

    want = vjp(lambda: 0.7)
    assert np.abs(want[1]).max() > 0
    for kw in ({}, {"stream": side}, {"stream": side.cuda_stream}):
        for a, b in zip(vjp(late, **kw), want):
            np.testing.assert_allclose(a, b, rtol=0, atol=1e-10 * max(1.0, np.abs(b).max()))
