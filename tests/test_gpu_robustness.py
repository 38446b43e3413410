"""Calls in the company of other work on the device: copies in flight, several handles and threads, little memory, long
chains, sectors that break down early, entries that are skipped or not finite."""
import numpy as np
import pytest

import ftlm_extended_hubbard_b200 as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lat,nu,nd", [((4, 3), 2, 2), ((4, 4), 3, 2)])
def test_momentum_blocks_built_while_copies_are_queued(gpu, lat, nu, nd):
    """A block's tables are on the device before its kernels read them, also with the copy engine busy: the default apply
    (the source lists, made from the tables when the block is created) against the hop scan, and the block's entries
    against those of an idle device."""
    torch = gpu
    p = F.HubbardParams(*lat, 1.0, -0.25, 6.0, 0.5)
    ks = [(0, 0), (1, 1), (lat[0] - 1, 0)]
    idle = F.Sector(p, nu, nd)
    want = [idle.orbit_block(*k).entries() for k in ks]
    host = torch.empty(1 << 28, dtype=torch.uint8, pin_memory=True)
    dev = torch.empty_like(host, device="cuda")
    side = torch.cuda.Stream()
    rng = np.random.default_rng(1)
    for k, (rep, absA) in zip(ks, want):
        s = F.Sector(p, nu, nd)
        with torch.cuda.stream(side):
            for _ in range(8):
                dev.copy_(host, non_blocking=True)
        o = s.orbit_block(*k)
        rep2, absA2 = o.entries()
        assert np.array_equal(rep, rep2) and np.array_equal(absA, absA2)
        x = rng.standard_normal(o.dim) + 1j * rng.standard_normal(o.dim)
        y = o.apply_host(x)
        o.set_apply_path(0)
        ref = o.apply_host(x)
        assert np.abs(y - ref).max() <= 1e-13 * max(1.0, np.abs(ref).max())
    torch.cuda.synchronize()
