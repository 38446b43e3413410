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


@pytest.mark.parametrize("method,R", [("plain", 1400), ("batched", 2800)])
def test_gradient_of_more_chains_than_a_store_holds(gpu, method, R):
    """60 vectors of 4,900 states for each of R chains are more than one 6 GB store: the gradient of all R chains is that of
    the two halves, each within a store, put together (ln Z is the log of a mean over chains, its gradient weighted by the
    means)."""
    lat = (4, 2)
    s = F.Sector(F.HubbardParams(*lat, 1.0, -0.2, 4.0, 1.0), 4, 4)
    op = F.Sector(F.HubbardParams(*lat, 0.0, 1.0, 0.0, 0.0), 4, 4)
    beta, M, seed, h = 2.0, 60, 11, R // 2
    kw = dict(op_tp=op, method=method, start="philox")
    lz, g = s.ftlm_grad(beta, R, M, seed, **kw)
    l1, g1 = s.ftlm_grad(beta, h, M, seed, **kw)
    l2, g2 = s.ftlm_grad(beta, h, M, seed + h * 100003, **kw)
    w1, w2 = np.exp(l1 - np.logaddexp(l1, l2)), np.exp(l2 - np.logaddexp(l1, l2))
    assert abs(lz - (np.logaddexp(l1, l2) - np.log(2.0))) <= 1e-11 * abs(lz)
    want = w1 * np.asarray(g1) + w2 * np.asarray(g2)
    assert np.abs(np.asarray(g) - want).max() <= 1e-9 * np.abs(want).max()
    F.api.batched_release()


def test_gradient_of_many_chains_with_short_rows(gpu):
    """Rows of one string, 12,870 of them, 160 vectors of each of 1,050 chains: more (row, vector) pairs than 31 bits
    number.  The gradient is that of five fifths of the chains put together; without down electrons dH/dU is zero."""
    s = F.Sector(F.HubbardParams(4, 4, 1.0, -0.2, 4.0, 0.0), 8, 0)
    op = F.Sector(F.HubbardParams(4, 4, 0.0, 1.0, 0.0, 0.0), 8, 0)
    beta, M = 0.5, 160
    lz, g = s.ftlm_grad(beta, 1050, M, 3, op_tp=op, start="philox")
    part = [s.ftlm_grad(beta, 210, M, 3 + 210 * 100003 * i, op_tp=op, start="philox") for i in range(5)]
    l = np.array([p[0] for p in part])
    w = np.exp(l - l.max())
    assert abs(lz - (l.max() + np.log(w.mean()))) <= 1e-11 * abs(lz)
    want = (w[:, None] * np.array([p[1] for p in part])).sum(0) / w.sum()
    assert g[0] == 0.0 and abs(g[2]) > 1e-3
    assert np.abs(np.asarray(g) - want).max() <= 1e-9 * np.abs(want).max()
    F.api.batched_release()


def test_gradient_with_an_operator_whose_row_does_not_fit(gpu):
    """A row of 12,870 strings fits shared memory, with a table of 240 different complex coefficients it does not: the
    derivative with respect to such an operator against the central difference of H + h * operator (1e-6, as the error of
    the difference at h = 1e-4)."""
    hops, pairs = F.build_hubbard_geometry(F.HubbardParams(4, 4, 1.0, -0.2, 0.0, 0.0))
    rng = np.random.default_rng(2)
    extra = []
    for i in range(16):
        for j in range(i):
            c = complex(0.1 + rng.random(), rng.standard_normal()) * 0.2
            extra += [F.SpinfulHopping(i, j, 1, c), F.SpinfulHopping(j, i, 1, c.conjugate())]

    def sector(h):
        more = [F.SpinfulHopping(e.from_, e.to, e.spin, h * e.coeff) for e in extra]
        return F.Sector(None, 0, 8, hops=list(hops) + more if h else hops, pairs=pairs, n_sites=16, U=0.0, V=0.0)

    op = F.Sector(None, 0, 8, hops=extra, pairs=pairs, n_sites=16, U=0.0, V=0.0)
    lz, g = sector(0.0).ftlm_grad(1.0, 2, 30, 5, op_tp=op, start="philox")
    h = 1e-4
    l1, l2 = (sector(x).ftlm(1.0, 2, 30, 5, start="philox")[0][0] for x in (h, -h))
    assert abs(g[2] - (l1 - l2) / (2 * h)) <= 1e-6 * max(1.0, abs(g[2]))


def test_momentum_block_lists_leave_the_memory_to_others(gpu):
    """With a gigabyte free a block of 207,000 states does without its lists (53 MB, more than a 32nd of what is free); the
    table form gives the list form's sums."""
    torch = gpu
    s = F.Sector(F.HubbardParams(4, 4, 1.0, -0.25, 6.0, 0.5), 4, 4)
    o = s.orbit_block(1, 2)
    rng = np.random.default_rng(6)
    x = rng.standard_normal(o.dim) + 1j * rng.standard_normal(o.dim)
    y = o.apply_host(x)
    F.api.batched_release()
    torch.cuda.empty_cache()
    taken = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    little = s.orbit_block(1, 2)
    used = free - torch.cuda.mem_get_info()[0]
    y2 = little.apply_host(x)
    del taken
    torch.cuda.empty_cache()
    assert used < 45 << 20  # 13 MB table, 8 MB of entries, 3 MB workspace, in blocks of 2 MB
    assert np.abs(y - y2).max() <= 1e-13 * np.abs(y).max()


def test_threads_share_a_fresh_handle(gpu):
    """Eight threads make the first calls of one handle at once: each gets the chains of a handle of its own."""
    import threading
    p = F.HubbardParams(3, 3, 1.0, -0.25, 8.0, 1.0)
    ref = F.Sector(p, 4, 4).batched_lanczos(4, 6, 3)
    for _ in range(5):
        s, out = F.Sector(p, 4, 4), [None] * 8
        ready = threading.Barrier(8)

        def work(i):
            ready.wait()
            out[i] = s.batched_lanczos(4, 6, 3)

        pool = [threading.Thread(target=work, args=(i,)) for i in range(8)]
        for t in pool:
            t.start()
        for t in pool:
            t.join()
        for o in out:
            assert all(np.array_equal(a, b) for a, b in zip(o, ref))


def test_handle_goes_while_its_call_is_in_flight(gpu):
    """A handle is dropped right after an asynchronous H v and another of the same shape takes its tables' place: both
    results are those of calls one at a time."""
    torch = gpu
    a, b = F.HubbardParams(4, 3, 1.0, -0.25, 8.0, 1.0), F.HubbardParams(4, 3, 0.5, 0.3, 2.0, 0.0)
    x = torch.randn(245025, dtype=torch.complex128, device="cuda")
    ref = []
    for p in (a, b):
        y = torch.empty_like(x)
        F.Sector(p, 4, 4).apply(x, y)
        torch.cuda.synchronize()
        ref.append(y)
    side = torch.cuda.Stream()
    for _ in range(10):
        out = [torch.empty_like(x) for _ in range(2)]
        torch.cuda.synchronize()
        for p, y in zip((a, b), out):
            s = F.Sector(p, 4, 4)
            for _ in range(20):
                s.apply(x, y, side.cuda_stream)
            s.close()
        torch.cuda.synchronize()
        assert torch.equal(out[0], ref[0]) and torch.equal(out[1], ref[1])


@pytest.mark.parametrize("path", [0, 3])
def test_threads_on_handles_of_different_sizes(gpu, path):
    """Two threads, each with a handle and a stream of its own and rows of 70 and 4,368 (one pass) or 924 and 11,440 strings
    (two passes): no call of one takes the shared memory that the other's kernel needs."""
    import threading
    torch = gpu
    shapes = [((4, 2), 4, 4), ((4, 4), 0, 5)] if path == 0 else [((4, 3), 6, 6), ((4, 4), 2, 7)]
    out, errors = [], []

    def work(lat, nu, nd):
        s = F.Sector(F.HubbardParams(*lat, 1.0, -0.25, 8.0, 1.0), nu, nd)
        s.set_apply_path(path)
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            x = torch.randn(s.dim(), dtype=torch.complex128, device="cuda")
            y, ref = torch.empty_like(x), torch.empty_like(x)
            s.apply(x, ref, st.cuda_stream)
            try:
                for _ in range(4000):
                    s.apply(x, y, st.cuda_stream)
            except F.FtlmError as e:
                errors.append(e)
            st.synchronize()
            out.append(torch.equal(y, ref))

    pool = [threading.Thread(target=work, args=c) for c in shapes]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not errors and out == [True, True]


@pytest.mark.parametrize("lat,nu,nd", [((3, 3), 4, 4), ((4, 2), 4, 4), ((4, 3), 4, 5)])
def test_chains_of_a_tuned_handle(gpu, lat, nu, nd):
    """Timing the H v variants leaves a small sector's chains in their fused kernel (the bits of an untuned handle) and a
    larger one's on planes, with the timed column slab (the dot products' order)."""
    p = F.HubbardParams(*lat, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0)
    s, t = F.Sector(p, nu, nd), F.Sector(p, nu, nd)
    t.autotune(2)
    a, b = s.lanczos(12, 5, start="philox"), t.lanczos(12, 5, start="philox")
    if s.dim() < 20000:
        assert all(np.array_equal(x, y) for x, y in zip(a[:2], b[:2]))
        assert np.array_equal(s.ftlm([0.5, 2.0], 3, 20, 5, start="philox")[0], t.ftlm([0.5, 2.0], 3, 20, 5, start="philox")[0])
    else:  # rounding grows by about two a step
        assert np.abs(a[0] - b[0]).max() <= 1e-11 * np.abs(a[0]).max()


def test_chains_keep_to_a_set_path(gpu):
    """A handle set to path 2 runs its chains on that path: the bits of the general recurrence on its own apply."""
    torch = gpu
    s = F.Sector(F.HubbardParams(4, 3, 1.0, -0.25, 8.0, 1.0), 4, 4)
    n = s.dim()
    for path in (1, 2):
        s.set_apply_path(path)
        a, b, _ = s.lanczos(8, 5, start="philox")
        a2, b2 = F.lanczos_tridiagonal(n, lambda x, y: s.apply(x, y), 8, 5, start="philox")[:2]
        assert np.array_equal(a, a2) and np.array_equal(b, b2)


def test_chains_that_end_early_do_no_further_work(gpu):
    """Without hopping a 4x4 (5,6) sector has the six levels 0, 8 .. 40, so its chains end after six steps, and 300 steps asked
    for take less time than 30 steps of a chain that goes on.  The chain is right, and so are complex64 chains and the
    gradient (d ln Z/dU of independent doublons is that of the levels' estimate)."""
    import time
    p = F.HubbardParams(4, 4, 0.0, 0.0, 8.0, 0.0)
    s, go = F.Sector(p, 5, 6), F.Sector(F.HubbardParams(4, 4, 1.0, -0.25, 8.0, 1.0), 5, 6)

    def seconds(h, steps):
        h.lanczos(2, 1, start="philox")
        t = time.perf_counter()
        out = h.lanczos(steps, 1, start="philox")
        return time.perf_counter() - t, out

    for _ in range(3):  # a busy machine may spoil a timing
        on, _ = seconds(go, 30)
        ended, (a, b, used) = seconds(s, 300)
        if ended < on:
            break
    assert ended < on
    assert used == a.size <= 8
    ritz = F.ritz_values(a, b[:used - 1], used)
    assert all(np.abs(ritz - v).min() <= 1e-8 for v in 8.0 * np.arange(6))
    A, B, u = s.batched_lanczos(3, 40, 1)
    assert np.abs(A[0, :5] - a[:5]).max() <= 1e-4 and np.isfinite(A).all()


def test_gradient_of_chains_that_end_early(gpu):
    """d ln Z/dU of the 4x3 (4,4) sector without hopping, chains on planes that end after five steps, against the central
    difference (1e-6 at h = 1e-4)."""
    def at(U):
        return F.Sector(F.HubbardParams(4, 3, 0.0, 0.0, U, 0.0), 4, 4)

    op = F.Sector(F.HubbardParams(4, 3, 0.0, 1.0, 0.0, 0.0), 4, 4)
    lz, g = at(4.0).ftlm_grad(0.7, 3, 60, 5, op_tp=op, start="philox")
    l1, l2 = (at(u).ftlm(0.7, 3, 60, 5, start="philox")[0][0] for u in (4.0 + 1e-4, 4.0 - 1e-4))
    assert abs(g[0] - (l1 - l2) / 2e-4) <= 1e-6 * max(1.0, abs(g[0])) and np.isfinite(g).all()


@pytest.mark.parametrize("k", [(0, 0), (2, 0)])
def test_momentum_block_values_that_almost_agree(gpu, k):
    """Hops of 1 and of 1 + 8e-15 are two values of the source lists: columns of H_K against the hop scan, to 9 ulp (a few
    products and square roots)."""
    s = F.Sector(F.HubbardParams(4, 3, 1.0, 1.0 + 8e-15, 4.0, 0.0), 2, 2)
    o = s.orbit_block(*k)
    for j in range(0, o.dim, 17):
        x = np.zeros(o.dim, complex)
        x[j] = 1.0
        o.set_apply_path(1)
        y = o.apply_host(x)
        o.set_apply_path(0)
        ref = o.apply_host(x)
        assert np.abs(y - ref).max() <= 2e-15 * np.abs(ref).max()


def test_handles_keep_the_vectors_of_one_chain(gpu):
    """After 32 chains at once (376 MB of vectors) a handle holds those of one chain; what the library keeps for the
    next call goes back with batched_release."""
    torch = gpu
    F.api.batched_release()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hold = [F.Sector(F.HubbardParams(4, 3, 1.0, -0.25, 8.0, 1.0), 4, 4) for _ in range(3)]
    for s in hold:
        s.ftlm([1.0], 32, 4, 1, start="philox")
    F.api.batched_release()
    assert free - torch.cuda.mem_get_info()[0] < 100 << 20  # tables, scalars and at most 12 MB of vectors each


def test_momentum_block_apply_of_entries_that_are_not_finite(gpu):
    """An infinite entry gives infinities and NaN where the hop scan has them: padding of the source lists adds nothing."""
    s = F.Sector(F.HubbardParams(4, 3, 1.0, -0.25, 4.0, 0.5), 2, 2)
    o = s.orbit_block(0, 0)
    rng = np.random.default_rng(8)
    for bad in (np.inf, -np.inf):
        x = rng.standard_normal(o.dim) + 1j * rng.standard_normal(o.dim)
        x[o.dim // 3] = bad
        o.set_apply_path(1)
        y = o.apply_host(x)
        o.set_apply_path(0)
        ref = o.apply_host(x)
        for part in (np.real, np.imag):
            a, b = part(y), part(ref)
            assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isinf(a), np.isinf(b))
            ok = np.isfinite(b)
            assert np.abs(a[ok] - b[ok]).max() <= 1e-12


@pytest.mark.parametrize("lat,nu,nd", [((3, 3), 4, 4), ((4, 3), 4, 4)])
def test_chains_of_numbers_that_are_not_finite(gpu, lat, nu, nd):
    """An interaction that is not a number gives a chain of as many alphas and betas as steps, fused and on planes, as the
    step-by-step recurrence does."""
    s = F.Sector(F.HubbardParams(*lat, 1.0, -0.25, float("nan"), 1.0), nu, nd)
    g = F.Sector(F.HubbardParams(*lat, 1.0, -0.25, float("nan"), 1.0), nu, nd)
    g.set_apply_path(1)
    a, b, used = s.lanczos(5, 1, start="philox")
    a2, b2, used2 = g.lanczos(5, 1, start="philox")
    assert used == used2 == 5 and a.size == a2.size == 5 and b.size == b2.size == 5
    assert np.isnan(b).all() and np.isnan(b2).all()


@pytest.mark.parametrize("lat,nu,nd,path", [((3, 3), 4, 4, 0), ((4, 2), 4, 4, 0), ((4, 4), 2, 2, 0), ((4, 3), 4, 4, 0), ((4, 3), 4, 4, 1),
                                            ((4, 3), 4, 4, 2), ((4, 3), 4, 4, 3)])
def test_entries_below_the_threshold_are_no_sources(gpu, lat, nu, nd, path):
    """Entries with |x|^2 < 1e-28 contribute nothing: a vector of such entries gives exact zeros, and beside others they leave
    the bits of the vector with zeros in their place (one pass and two, a row of the block and other rows)."""
    torch = gpu
    s = F.Sector(F.HubbardParams(*lat, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0), nu, nd)
    s.set_apply_path(path)
    gen = torch.Generator(device="cuda").manual_seed(5)
    small = torch.randn(s.dim(), dtype=torch.complex128, device="cuda", generator=gen)
    small = 9e-15 * small / small.abs()
    y, ref = torch.empty_like(small), torch.empty_like(small)
    s.apply(small, y)
    assert not y.any()
    for every in (2, 37, s.dim()):
        x, x0 = small.clone(), torch.zeros_like(small)
        x[::every] = x0[::every] = 1.0 + 0.5j
        s.apply(x, y)
        s.apply(x0, ref)
        assert torch.equal(y, ref) and ref.any()


@pytest.mark.parametrize("lat,nu,nd,k", [((4, 3), 3, 3, (1, 1)), ((3, 3), 4, 2, (0, 0)), ((4, 4), 3, 2, (2, 1))])
@pytest.mark.parametrize("path", [0, 1])
def test_entries_below_the_threshold_in_a_momentum_block(gpu, lat, nu, nd, k, path):
    """The same in a momentum block, from its source lists and by the hop scan."""
    torch = gpu
    o = F.Sector(F.HubbardParams(*lat, 1.0, -0.25, 6.0, 0.5), nu, nd).orbit_block(*k)
    o.set_apply_path(path)
    gen = torch.Generator(device="cuda").manual_seed(6)
    small = torch.randn(o.dim, dtype=torch.complex128, device="cuda", generator=gen)
    small = 9e-15 * small / small.abs()
    y, ref = torch.empty_like(small), torch.empty_like(small)
    o.apply(small, y)
    assert not y.any()
    for every in (2, 37, o.dim):
        x, x0 = small.clone(), torch.zeros_like(small)
        x[::every] = x0[::every] = 1.0 + 0.5j
        o.apply(x, y)
        o.apply(x0, ref)
        assert torch.equal(y, ref) and ref.any()


@pytest.mark.parametrize("nu,nd", [(0, 8), (8, 0), (8, 1), (1, 5), (5, 1), (4, 1), (0, 4)])
def test_default_apply_of_thin_sectors(gpu, nu, nd):
    """Sectors with few strings of one species: the default H v is the faster of the one pass and the generic kernel (to 30 %,
    which a wrong choice exceeds by far), and gives its sums (1e-13 of the largest)."""
    torch = gpu
    s = F.Sector(F.HubbardParams(4, 4, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0), nu, nd)
    x = torch.randn(s.dim(), dtype=torch.complex128, device="cuda")
    y, ref = torch.empty_like(x), torch.empty_like(x)

    def us(path, out):
        s.set_apply_path(path)
        best = 1e9
        for _ in range(5):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            s.apply(x, out)
            a.record()
            for _ in range(50):
                s.apply(x, out)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 20.0)
        return best

    for _ in range(3):  # a busy machine may spoil a timing
        generic, default = us(1, ref), us(0, y)
        if default <= 1.3 * generic:
            break
    assert default <= 1.3 * generic
    assert (y - ref).abs().max() <= 1e-13 * ref.abs().max()


@pytest.mark.parametrize("lat,nu,nd", [((4, 4), 0, 8), ((4, 4), 8, 0), ((4, 4), 6, 0), ((4, 4), 8, 1), ((3, 3), 3, 3), ((4, 3), 4, 1),
                                       ((4, 4), 0, 5), ((3, 3), 4, 4)])
def test_chain_of_a_small_or_thin_sector(gpu, lat, nu, nd):
    """One chain runs no slower than the general recurrence on the generic H v (to 15 %; the wrong one of the three forms
    costs up to five times), and gives its alpha (rounding grows by about two a step)."""
    import time
    s = F.Sector(F.HubbardParams(*lat, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0), nu, nd)

    def run(path):
        s.set_apply_path(path)
        best = 1e9
        for _ in range(6):
            t = time.perf_counter()
            a = s.lanczos(40, 3, start="philox")[0]
            best = min(best, time.perf_counter() - t)
        return best, a

    for _ in range(3):  # a busy machine may spoil a timing
        (general, a1), (default, a0) = run(1), run(0)
        if default <= 1.15 * general:
            break
    assert default <= 1.15 * general
    assert np.abs(a0[:8] - a1[:8]).max() <= 1e-11 * np.abs(a1).max()


def test_column_pass_by_items_and_on_the_persistent_grid(gpu):
    """5x3 (3,6): slabs of 256 and 128 columns run one block per item, 512 columns the persistent grid (a plane has 9,100, 18,200
    and 4,550 items). One chain with each, against the general recurrence (rounding grows by about two a step)."""
    from ftlm_extended_hubbard_b200 import _lib
    s = F.Sector(F.HubbardParams(5, 3, 1.0, -0.25, 8.0, 1.0, 0.1, 0.0), 3, 6)
    s.set_apply_path(1)
    a1, b1, _ = s.lanczos(8, 3, start="philox")
    s.set_apply_path(0)
    for v in (0, 1, 2):
        _lib.call("ftlm_gpu_set_cols_variant", s.handle, v)
        a, b, _ = s.lanczos(8, 3, start="philox")
        assert np.abs(a - a1).max() <= 1e-12 * np.abs(a1).max() and np.abs(b - b1).max() <= 1e-12 * np.abs(b1).max()


@pytest.mark.parametrize("lat,nu,nd,method", [((3, 3), 3, 2, "plain"), ((3, 3), 4, 5, "batched"), ((4, 3), 4, 4, "plain"), ((4, 3), 4, 4, "batched")])
def test_gradient_of_an_odd_number_of_planes(gpu, lat, nu, nd, method):
    """25 vectors of each of three or five chains: an odd number of planes, of which the operator's row pass takes two at a
    time.  The gradient is that of the chains one by one (complex64: two by two and one) put together."""
    s = F.Sector(F.HubbardParams(*lat, 1.0, -0.2, 4.0, 1.0), nu, nd)
    op = F.Sector(F.HubbardParams(*lat, 0.0, 1.0, 0.0, 0.0), nu, nd)
    kw = dict(op_tp=op, method=method, start="philox")
    R, M, beta, seed = (3, 25, 1.5, 7) if method == "plain" else (5, 25, 1.5, 7)
    parts = [(r, 1) for r in range(R)] if method == "plain" else [(0, 2), (2, 2), (4, 1)]
    lz, g = s.ftlm_grad(beta, R, M, seed, **kw)
    p = [(n,) + s.ftlm_grad(beta, n, M, seed + r * 100003, **kw) for r, n in parts]
    w = np.array([n * np.exp(l - lz) for n, l, _ in p]) / R
    tol = 1e-10 if method == "plain" else 1e-6
    assert abs(w.sum() - 1.0) <= tol
    want = (w[:, None] * np.array([q[2] for q in p])).sum(0) / w.sum()
    assert np.abs(np.asarray(g) - want).max() <= 10 * tol * np.abs(want).max()
