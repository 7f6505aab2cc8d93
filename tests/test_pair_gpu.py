"""Two steps in one launch against single steps, bit for bit: the pair runs
the same per-node arithmetic and rounding, so populations, moments and sums
agree exactly over every boundary, wrap, ragged size and storage it takes."""
import ctypes

import numpy as np
import pytest

import cases as C

pytestmark = pytest.mark.gpu

# sizes around the 32 x 8 tiles of small lattices: smaller than one, a whole
# number, one node more or less, several ragged ones
SIZES = [(3, 3), (5, 40), (63, 15), (64, 16), (65, 17), (66, 18), (129, 33), (200, 47)]


def porous(nx, ny, **kw):
    """Scattered obstacles of every local boundary among fluid nodes (few
    enough for pairs), a force field and a Brinkman field."""
    c = C.taylor_green(nx, ny, nu=0.05, **kw)
    r = np.random.default_rng(3)
    c["flags"][:] = r.choice([C.FLUID, C.CYLINDER, C.HALFWAY_BB, C.MOVING_WALL_BB, C.BOUNCE_BACK], (ny, nx),
                             p=[0.997, 0.0006, 0.0006, 0.0006, 0.0012])
    c["wall_u"] = (0.03, 0.01)
    c["force"] = 1e-5 * r.standard_normal((2, ny, nx))
    c["gamma"] = r.uniform(0.0, 0.3, (ny, nx)).astype(np.float32)
    return c


def corners(nx, ny, **kw):
    c = C.channel(nx, ny, inlet="parabolic", outlet="zouhe_p", **kw)
    c["flags"][-1, 0], c["flags"][0, 0] = C.CORNER_TOP_LEFT, C.CORNER_BOTTOM_LEFT
    return c


def regularized(nx, ny, **kw):
    c = C.cavity_regularized(nx, ny, **kw)
    c["flags"][c["flags"] == C.REGULARIZED_BOUNCE_BACK_CORNER] = C.REGULARIZED_BOUNCE_BACK
    return c


def open_box(nx, ny, **kw):
    """Fluid up to non-periodic edges: every edge node reads the edge store."""
    return C.base(nx, ny, kw.pop("op"), 0.05, **kw)


FLOWS = {"vortex": C.taylor_green, "cavity": C.cavity_moving_wall, "zouhe": C.cavity_zouhe, "poiseuille": C.poiseuille,
         "corners": corners, "regularized": regularized, "porous": porous, "open": open_box}


def lattices(c, storage, count=2):
    out = [C.make_lattice(c, storage=storage) for _ in range(count)]
    for L in out:
        if "gamma" in c:
            L.set_brinkman(c["gamma"])
    return out


def same(A, B):
    assert A.t == B.t
    np.testing.assert_array_equal(A.populations(), B.populations())
    ra, ua, sa = A.moments()
    rb, ub, sb = B.moments()
    np.testing.assert_array_equal(ra, rb)
    np.testing.assert_array_equal(ua, ub)
    np.testing.assert_array_equal(sa, sb)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("flow", sorted(FLOWS))
def test_pairs_equal_single_steps(flow, size):
    import lbmx
    for k, (op, storage) in enumerate([(C.BGK, 0), (C.MRT, 1), (C.CM, 0), (C.CM, 2)]):
        c = C.random_state(FLOWS[flow](size[0], size[1], op=op), seed=k)
        A, B = lattices(c, storage)
        # even and odd starts, odd counts, moments stored by a pair and by a single step
        for n in (2, 5, 1, 4):
            A.step(n)
            for i in range(n):
                B.step(1, flags=lbmx.STEP_STORE_MOMENTS if i == n - 1 else 0)
            same(A, B)


@pytest.mark.parametrize("flow", ["porous", "corners", "cavity"])
@pytest.mark.parametrize("nx,ny,op,storage", [
    (651, 130, C.MRT, 0),    # 32 x 16 tiles
    (650, 129, C.BGK, 1),
    (1301, 531, C.MRT, 0),   # 64 x 12
    (1281, 496, C.CM, 0),    # 64 x 16
    (1300, 701, C.BGK, 1),
    (2001, 901, C.MRT, 1),   # 64 x 20
])
def test_larger_tiles(flow, nx, ny, op, storage):
    import lbmx
    A, B = lattices(C.random_state(FLOWS[flow](nx, ny, op=op), seed=9), storage)
    for n in (4, 3):
        A.step(n, flags=lbmx.STEP_STORE_MOMENTS | lbmx.STEP_SUMS)
        for _ in range(n):
            B.step(1)
        same(A, B)


@pytest.mark.parametrize("flags", [0, 1, 9, 3])
def test_series_of_pairs(flags):
    """Per-step sums through pinned memory (pairs) and pageable memory (single steps)."""
    import torch
    import lbmx
    c = C.random_state(C.cavity_moving_wall(200, 47, op=C.MRT), seed=4)
    A, B = lattices(c, 0)
    width = 4 if flags & lbmx.STEP_KINETIC_ENERGY else 3
    for n in (6, 3, 4):
        got = torch.zeros((n, width), dtype=torch.float64).pin_memory()
        A._check(A.lib.lbmx_step_sums(A.h, n, flags, got.data_ptr()))
        want = B.step_sums(n, flags)
        A.synchronize()
        np.testing.assert_array_equal(got.numpy(), want)
        np.testing.assert_array_equal(A.moments()[2], B.moments()[2])
        A.step(1, flags=lbmx.STEP_SUMS)
        B.step(1, flags=lbmx.STEP_SUMS)
        np.testing.assert_array_equal(A.moments()[2], B.moments()[2])


def test_mass_of_a_large_lattice_near_rest():
    """More than 2^16 units a warp, none of whose sums calls for a total
    before the end: 2 CTAs x 8 warps on 152 SMs, FP32 CM."""
    import torch
    import lbmx
    n = 18560
    free, total = torch.cuda.mem_get_info()
    if free < 72 * n * n + 30 * n * n + total * 3 // 4:
        pytest.skip("not enough device memory for a lattice of this size with its second buffer")
    rho = torch.ones((n, n), device="cuda")
    u = torch.zeros((2, n, n), device="cuda")
    torch.cuda.synchronize()
    L = lbmx.Lattice(n, n, op=lbmx.CM, omega=1.2, periodic=(True, True))
    sums = []
    for calls in ([2], [1, 1]):
        L.init(rho, u)
        for k in calls:
            L.step(k)
        s = (ctypes.c_double * 3)()
        L._check(L.lib.lbmx_moments(L.h, None, None, s))
        sums.append(list(s))
    L.close()
    del rho, u
    torch.cuda.empty_cache()
    assert sums[0] == sums[1]
    assert abs(sums[0][0] - n * n) < 1e-6 * n * n


def test_flags_changed_between_pairs():
    """A half-way wall turned bounce-back reads the edge-store values its
    nodes had before, whichever buffers the pairs left the state in."""
    c = C.random_state(C.cavity_moving_wall(70, 37, op=C.BGK), seed=5)
    d = C.cavity_zouhe(70, 37, op=C.BGK)["flags"]
    A, B = lattices(c, 0)
    for fl in (c["flags"], d, c["flags"], d):
        for L in (A, B):
            L.set_flags(fl)
        A.step(6)
        for _ in range(6):
            B.step(1)
        same(A, B)


def test_steps_captured_into_a_graph():
    """Captured steps stay in one buffer, so that a graph can be replayed:
    six replays of two steps, after steps taken in pairs."""
    import torch
    stream = torch.cuda.Stream()
    c = C.random_state(C.cavity_moving_wall(96, 40, op=C.MRT), seed=6)
    A = C.make_lattice(c, stream=stream.cuda_stream)
    B = C.make_lattice(c)
    A.step(6, flags=0)
    A.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        A.step(2, flags=0)
    with torch.cuda.stream(stream):
        for _ in range(6):
            graph.replay()
    A.step(2)  # (moments of the state the replays left)
    for _ in range(6 + 12 + 2):
        B.step(1)
    ra, ua, _ = A.moments()
    rb, ub, _ = B.moments()
    np.testing.assert_array_equal(ra, rb)
    np.testing.assert_array_equal(ua, ub)


def test_direct_steps_between_replays():
    """After a capture the state stays in the graph's buffers: replays and
    direct steps in turn, then a fresh state."""
    import torch
    stream = torch.cuda.Stream()
    c = C.random_state(C.cavity_moving_wall(96, 40, op=C.MRT), seed=6)
    A = C.make_lattice(c, stream=stream.cuda_stream)
    B = C.make_lattice(c)
    A.step(2, flags=0)
    A.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        A.step(2, flags=0)

    def replay(n):
        with torch.cuda.stream(stream):
            for _ in range(n):
                graph.replay()

    def check(steps):
        for _ in range(steps):
            B.step(1)
        for x, y in zip(A.moments(), B.moments()):
            np.testing.assert_array_equal(x, y)

    replay(3)
    A.step(2)
    check(2 + 6 + 2)
    replay(1)
    A.step(4)
    check(2 + 4)
    for L in (A, B):
        L.init(np.asarray(c["rho"], np.float32), np.asarray(c["u"], np.float32))
    replay(2)
    A.step(2)
    check(4 + 2)


def test_captured_averages_pre_pass_replayed_alone():
    """CM_OPT with lagged averages: only the first of the two captured steps
    has a pre-pass, and each of its replays computes the same averages as a
    direct step from that state."""
    import torch
    import lbmx
    stream = torch.cuda.Stream()
    c = C.random_state(C.cavity_moving_wall(96, 40, op=C.CM_OPT), seed=8)
    A = C.make_lattice(c, options=lbmx.OPTION_LAGGED_AVERAGES, stream=stream.cuda_stream)
    B = C.make_lattice(c)
    first, second = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    for graph in (first, second):
        with torch.cuda.graph(graph, stream=stream):
            A.step(1)
    for _ in range(3):
        with torch.cuda.stream(stream):
            first.replay()
        B.step(1)
        avg = B.averages()
        np.testing.assert_allclose(A.averages(), avg, rtol=1e-6)
        with torch.cuda.stream(stream):
            second.replay()
        B.set_averages(avg)  # the second step lags: the averages of the first
        B.step(1)
        for x, y in zip(A.moments(), B.moments()):
            np.testing.assert_allclose(x, y, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("flow", ["open", "corners", "cavity"])
def test_steps_after_a_batch(flow):
    """A lattice that left its batches (in odd numbers of steps, the edge
    store included) goes on as one that was never in any."""
    import lbmx
    c = C.random_state(FLOWS[flow](129, 33, op=C.MRT), seed=2)
    A, B = lattices(c, 0)
    A.step(4)
    one, two = lbmx.Batch([A]), lbmx.Batch([A])
    one.step(3)
    one.close()
    A.step(3)
    two.step(4)
    two.close()
    A.step(6)
    for _ in range(20):
        B.step(1)
    same(A, B)


def test_a_lattice_that_left_its_batch_is_as_fast_as_before():
    """Two steps per launch again (4096^2 FP32: 1.8 times a single step's
    rate; half of that gain is asked for)."""
    import torch
    import lbmx
    stream = torch.cuda.Stream()
    best = []
    for batched in (False, True):
        L = lbmx.Lattice(4096, 4096, op=lbmx.MRT, omega=1.2, periodic=(True, True), stream=stream.cuda_stream)
        L.init(np.ones((4096, 4096), np.float32), np.zeros((2, 4096, 4096), np.float32))
        if batched:
            b = lbmx.Batch([L])
            b.step(2)
            b.close()
        times = []
        for _ in range(4):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record(stream)
            L.step(40, flags=0)
            e[1].record(stream)
            L.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        best.append(min(times))
        L.close()
    assert best[1] < 1.4 * best[0], best


def test_spare_buffers_make_way_for_a_new_lattice():
    """On a full device the second buffer of one lattice is given back for
    the allocations of another, which fit without it; the first goes on."""
    import torch
    import lbmx
    n = 4096  # 0.6 GB a buffer; given back: that less 0.2 GB of staging

    def start():
        L = lbmx.Lattice(n, n, op=lbmx.MRT, omega=1.3, periodic=(True, True))
        L.init(rho, u)
        return L

    r = np.random.default_rng(4)
    rho = (1 + 0.01 * r.standard_normal((n, n))).astype(np.float32)
    u = (0.01 * r.standard_normal((2, n, n))).astype(np.float32)
    B = start()
    for _ in range(2 + 3 + 2):
        B.step(1)
    want = B.moments()
    B.close()
    torch.cuda.empty_cache()
    A = start()
    A.step(2)
    A.synchronize()
    free = torch.cuda.mem_get_info()[0]
    full = torch.empty(free - (128 << 20), dtype=torch.uint8, device="cuda")
    try:
        C2 = lbmx.Lattice(2048, 2048, op=lbmx.MRT, omega=1.3, periodic=(True, True))  # 0.25 GB
    finally:
        del full
        torch.cuda.empty_cache()
    C2.close()
    A.step(3)
    A.step(2)
    for x, y in zip(A.moments(), want):
        np.testing.assert_array_equal(x, y)
    # and its init fields have their own staging now
    A.init(rho, u)
    A.step(7)
    for x, y in zip(A.moments(), want):
        np.testing.assert_array_equal(x, y)


def test_single_buffer_option():
    import torch
    import lbmx
    n = 2048
    used = []
    torch.cuda.synchronize()
    for options in (0, lbmx.OPTION_SINGLE_BUFFER):
        before = torch.cuda.mem_get_info()[0]
        L = lbmx.Lattice(n, n, op=lbmx.BGK, omega=1.3, periodic=(True, True), options=options)
        used.append(before - torch.cuda.mem_get_info()[0])
        L.close()
    # 36 bytes a node of second buffer against 12 of staging
    assert used[0] - used[1] > 20 * n * n, used
    c = C.random_state(C.cavity_moving_wall(70, 37, op=C.BGK), seed=5)
    A, B = C.make_lattice(c), C.make_lattice(c, options=lbmx.OPTION_SINGLE_BUFFER)
    for n in (2, 3, 4):
        A.step(n)
        B.step(n)
        same(A, B)


def test_adjoint_segment_makes_way():
    """The segment kept by a forward run is given back to another object's
    allocation and recomputed by the backward run, to the same gradient."""
    import torch
    import lbmx
    nx = ny = 1024  # 36 MB a state, 15 of them in the segment
    r = np.random.default_rng(7)
    rho, u = np.ones((ny, nx), np.float32), (0.01 * r.standard_normal((2, ny, nx))).astype(np.float32)
    gamma = (0.1 * r.random((ny, nx))).astype(np.float32)
    w = np.zeros((3, ny, nx), np.float32)
    w[1] = r.random((ny, nx))
    a = lbmx.Adjoint(nx, ny, op=lbmx.CM, omega=1.2, periodic=(True, True), checkpoint_every=16)
    a.set_state(rho, u)
    a.set_gamma(gamma)
    a.set_objective(w, 1)
    a.forward(20)
    want, scalars = a.backward()
    a.forward(16)
    a.forward(20)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    full = torch.empty(free - (128 << 20), dtype=torch.uint8, device="cuda")
    try:
        L = lbmx.Lattice(2048, 2048, op=lbmx.MRT, omega=1.3, periodic=(True, True))
    finally:
        del full
        torch.cuda.empty_cache()
    L.close()
    got, s = a.backward()
    np.testing.assert_array_equal(got, want)
    assert s == scalars
