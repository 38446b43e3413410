"""The kernels that small sectors take by default, at the sizes where their mapping changes: strings shorter than a warp
and just past its width, the fused chains' staging of a block of rows, momentum blocks in both source forms."""
import numpy as np
import pytest

import ftlm_extended_hubbard_b200 as F
import oracle as O

pytestmark = pytest.mark.gpu

# (lattice, n_up, n_dn): rows of 1, 9, 16 < 32 strings, 36, 66, 126; one row; a phase in one and in both directions
SECTORS = [((3, 3, 1.0, -0.25, 8.0, 1.0, 0.0, 0.0), 4, 0), ((3, 3, 1.0, 0.3, 2.0, 0.7, 0.1, 0.0), 4, 1),
           ((4, 4, 1.0, -0.25, 8.0, 1.0, 0.1, 0.2), 2, 1), ((3, 3, 1.0, 0.137, 8.0, 1.0, 0.0, 0.3), 5, 2),
           ((4, 3, 1.0, -0.25, 4.0, 1.0, 0.1, 0.2), 3, 2), ((3, 3, 1.0, -0.25, 8.0, 1.0, 0.1, 0.2), 4, 4),
           ((3, 3, 1.0, -0.25, 8.0, 1.0, 0.0, 0.0), 0, 4), ((4, 2, 1.0, 0.0, 8.0, 1.0, 0.0, 0.0), 4, 4)]


@pytest.mark.parametrize("case", SECTORS, ids=lambda c: f"{c[0][0]}x{c[0][1]}_{c[1]}{c[2]}")
def test_default_apply_of_small_sectors(gpu, case):
    """One pass (the default) against the oracle: sums of at most 100 products, 1e-13 of the largest; entries below the
    skip threshold and exact zeros among the sources, in the row and in other rows."""
    lat, nu, nd = case
    s, o = F.Sector(F.HubbardParams(*lat), nu, nd), O.OracleSector(*lat, nu, nd)
    rng = np.random.default_rng(nu * 17 + nd)
    x = rng.standard_normal(s.dim()) + 1j * rng.standard_normal(s.dim())
    x[rng.random(s.dim()) < 0.1] = 0.0
    x[rng.random(s.dim()) < 0.1] = 5e-15
    y, ref = s.apply_host(x), o.apply(x, mode=0)
    assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("case", SECTORS, ids=lambda c: f"{c[0][0]}x{c[0][1]}_{c[1]}{c[2]}")
def test_fused_chains_follow_the_general_recurrence(gpu, case):
    """The first steps of fused complex128 chains (set_apply_path(1) runs the general recurrence) and of complex64
    chains: rounding grows by about a factor of two a step from 1e-15 (1e-7 in complex64)."""
    lat, nu, nd = case
    s, g = F.Sector(F.HubbardParams(*lat), nu, nd), F.Sector(F.HubbardParams(*lat), nu, nd)
    g.set_apply_path(1)
    steps = min(8, s.dim() - 1)
    for start in ("reference", "philox"):
        a, b, u = s.lanczos(steps, 5, start=start)
        a2, b2, u2 = g.lanczos(steps, 5, start=start)
        n = min(u, u2)  # an exhausted Krylov space may end a step apart
        assert abs(u - u2) <= 1
        assert np.abs(a[:n] - a2[:n]).max() <= 1e-11 * max(1.0, np.abs(a2).max())
    A, B, used = F.api.lanczos_sectors([s, g], 3, steps, 5, "philox")
    assert np.array_equal(A[:3], A[3:]) and np.array_equal(used[:3], used[3:])
    assert np.abs(A[0, :n] - a[:n]).max() <= 1e-11 * max(1.0, np.abs(a).max())


@pytest.mark.parametrize("nu,nd,M", [(4, 4, 20), (3, 4, 12)])
def test_sweep_sectors_fused_or_alone(gpu, nu, nd, M):
    """A 3x3 sector's complex64 estimate alone (its own call) and within the sweep's fused launch: the same FP32 chains,
    FP64 sums in another order."""
    p = F.HubbardParams(3, 3, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0)
    T = np.array([0.3, 1.0])
    r = F.grand_canonical_sweep(p, 5, M, 9, T, np.array([0.0]), method="batched")
    lz, e = F.Sector(p, nu, nd).batched_ftlm(1.0 / T, 5, M, 9)
    assert np.abs(lz - r.lnz_sector[nu * 10 + nd]).max() <= 1e-9 * np.abs(lz).max()
    assert np.abs(e - r.e_sector[nu * 10 + nd]).max() <= 1e-9 * np.abs(e).max()


@pytest.mark.parametrize("case", [((5, 3, 1.0, -0.25, 6.0, 0.5, 0.0, 0.0), 3, 2, (2, 1)), ((4, 3, 1.0, 0.3, 6.0, 0.5, 0.0, 0.0), 1, 1, (1, 2)),
                                  ((2, 2, 1.0, -0.25, 6.0, 0.5, 0.0, 0.0), 2, 2, (0, 0)), ((4, 4, 1.0, -0.25, 6.0, 0.5, 0.0, 0.0), 8, 1, (2, 2))],
                         ids=lambda c: f"{c[0][0]}x{c[0][1]}_{c[1]}{c[2]}")
def test_momentum_block_source_lists(gpu, case):
    """H_K v from the source lists (path 1) against the hop scan (path 0): lattices of 15, 12, 4 and 16 translations,
    blocks of a few states, stabilisers of several sizes; tiny entries are skipped sources."""
    lat, nu, nd, k = case
    o = F.Sector(F.HubbardParams(*lat), nu, nd).orbit_block(*k)
    rng = np.random.default_rng(3)
    x = rng.standard_normal(o.dim) + 1j * rng.standard_normal(o.dim)
    x[rng.random(o.dim) < 0.1] = 5e-15
    y = o.apply_host(x)
    o.set_apply_path(0)
    ref = o.apply_host(x)
    assert np.abs(y - ref).max() <= 1e-13 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("case", [((3, 3, 1.0, -0.25, 8.0, 1.0, 0.0, 0.0), 4, 4), ((3, 3, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0), 5, 4),
                                  ((3, 3, 1.0, 0.3, 2.0, 0.7, 0.1, 0.0), 4, 1), ((4, 2, 1.0, 0.3, 8.0, 1.0, 0.0, 0.0), 3, 4),
                                  ((3, 3, 1.0, -0.25, 8.0, 1.0, 0.2, 0.0), 3, 6), ((3, 3, 1.0, -0.25, 8.0, 1.0, 0.1, 0.2), 3, 2)],
                         ids=lambda c: f"{c[0][0]}x{c[0][1]}_{c[1]}{c[2]}_{c[0][6]}")
def test_fused_chains_in_both_list_forms(gpu, case):
    """Packed up lists (real hops, one phase) and the general list, staged whole and by rows, rows of 9 to 126 strings
    with a last group of 4 to 30: complex128 within 1e-11 of the general recurrence over 6 steps, complex64 within 1e-5
    over 4 (4e-7 from sums of 40 products, doubled a step)."""
    lat, nu, nd = case
    s, g = F.Sector(F.HubbardParams(*lat), nu, nd), F.Sector(F.HubbardParams(*lat), nu, nd)
    g.set_apply_path(1)
    a, _, _ = s.lanczos(6, 5, start="philox")
    a2, _, _ = g.lanczos(6, 5, start="philox")
    scale = max(1.0, np.abs(a2).max())
    assert np.abs(a - a2).max() <= 1e-11 * scale
    A = s.batched_lanczos(3, 4, 5)[0]
    assert np.abs(A[0, :4] - a2[:4]).max() <= 1e-5 * scale


def test_skip_rule_over_calls_of_one_sector(gpu):
    """The two passes agree on each call's own input: with and without entries below the skip threshold in turn, launched and
    replayed from a graph, one handle gives the bits of a fresh handle (an input with such an entry takes the filter)."""
    import torch
    p = F.HubbardParams(4, 3, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0)
    s = F.Sector(p, 4, 5)
    s.set_apply_path(3)
    gen = torch.Generator(device="cuda").manual_seed(4)
    plain = torch.randn(s.dim(), dtype=torch.complex128, device="cuda", generator=gen)
    small = plain.clone()
    small[::7] = 5e-15
    ref = []
    for v in (plain, small):
        f = F.Sector(p, 4, 5)
        f.set_apply_path(3)
        y = torch.empty_like(v)
        f.apply(v, y)
        ref.append(y)
    x, y = plain.clone(), torch.empty_like(plain)
    s.apply(x, y)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        s.apply(x, y, torch.cuda.current_stream().cuda_stream)
    for k in (1, 0, 1, 1, 0, 0, 1):
        x.copy_(small if k else plain)
        for run in (lambda: s.apply(x, y), graph.replay):
            y.zero_()
            run()
            assert torch.equal(y, ref[k])


@pytest.mark.parametrize("lat,nu,nd", [((4, 3), 3, 4), ((4, 3), 4, 5), ((4, 4), 2, 3), ((5, 3), 4, 4)])
def test_calls_in_flight_keep_their_order(gpu, lat, nu, nd):
    """Two-pass calls launched ahead of one another (67,200 to 1,863,225 states), each on the result of the one before with
    an elementwise kernel between, on the default stream and on another one: the bits of the same calls one at a time."""
    import torch
    s = F.Sector(F.HubbardParams(*lat, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0), nu, nd)
    s.set_apply_path(3)
    gen = torch.Generator(device="cuda").manual_seed(nu)
    x0 = torch.randn(s.dim(), dtype=torch.complex128, device="cuda", generator=gen)

    def chain(stream, wait):
        with torch.cuda.stream(stream):
            x, y = x0.clone(), torch.empty_like(x0)
            for k in range(24):
                s.apply(x, y, stream.cuda_stream)
                if wait:
                    torch.cuda.synchronize()
                if k % 3:
                    y.mul_(0.05)
                x, y = y, x
        torch.cuda.synchronize()
        return x

    ref = chain(torch.cuda.default_stream(), True)
    for stream in (torch.cuda.default_stream(), torch.cuda.Stream()):
        for _ in range(3):
            assert torch.equal(chain(stream, False), ref)
