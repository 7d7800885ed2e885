"""The vector loops of the folds and copies where they can go wrong: every pair of 8-bit float
codes and every 16-bit code against awkward partners, every rank count that has a loop of its own,
blocks that end inside a vector, buffers at any element offset. Compared bit for bit with the host
schedules (hxccl_b200.ops.oracle)."""
import ctypes as C

import numpy as np
import pytest

from hxccl_b200 import _lib as L
from hxccl_b200.ops import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def worlds():
    from hxccl_b200.ops.world import World

    made = {}

    def get(n):
        if n not in made:
            made[n] = World(n, window_mb=8, wait_ms=20000)
        return made[n]

    yield get
    for w in made.values():
        w.close()


def dev(a, shift=0):
    """`a` on the GPU, `shift` bytes behind a 256-byte boundary"""
    raw = torch.zeros(a.nbytes + 256, dtype=torch.uint8, device="cuda")
    out = raw[shift:shift + a.nbytes]
    out.copy_(torch.from_numpy(a.view(np.uint8).copy()))
    return out


def back(t, dt):
    return t.cpu().numpy().view(oracle.raw_dtype(dt))


def pairs(dt):
    if L.DTYPE_SIZE[dt] == 1:
        a, b = np.meshgrid(np.arange(256, dtype=np.uint8), np.arange(256, dtype=np.uint8))
        return a.ravel().copy(), b.ravel().copy()
    special = np.array([0, 1, 2, 0x3ff, 0x400, 0x7bff, 0x7c00, 0x7c01, 0x7e00, 0x7f7f, 0x7f80, 0x7f81, 0x7fff, 0x3c00, 0x3f80, 0x3555],
                       dtype=np.uint16)
    special = np.concatenate([special, special | 0x8000])
    codes = np.arange(65536, dtype=np.uint16)
    return np.tile(codes, len(special)), np.repeat(special, len(codes))


@pytest.mark.parametrize("dt", [L.FLOAT8E4M3, L.FLOAT8E5M2, L.FLOAT16, L.BFLOAT16])
def test_every_code_of_the_narrow_types(worlds, dt):
    w = worlds(2)
    a, b = pairs(dt)
    for op in (L.SUM, L.PROD, L.MAX):
        for variant, order in ((1, 0), (1, 1), (6, 0)):
            w.tune(variant=variant, exact=True)
            send = [dev(a), dev(b)]
            recv = [torch.zeros_like(s) for s in send]
            w.all_reduce(send, recv, len(a), dt, op=op, order=order)
            torch.cuda.synchronize()
            want = oracle.allreduce([a, b], dt, op, order=order)
            for r in range(2):
                assert np.array_equal(back(recv[r], dt), want[r]), (dt, op, variant, order, r)
    w.tune(variant=0, exact=True)


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 8])
def test_rank_counts_block_ends_and_offsets(worlds, n):
    w = worlds(n)
    rng = np.random.default_rng(n)
    for dt in (L.FLOAT32, L.BFLOAT16, L.FLOAT8E4M3, L.INT32):
        es = L.DTYPE_SIZE[dt]
        for op in (L.SUM, L.AVG, L.MAX):
            # blocks shorter than a vector, ends inside vectors, several runs per warp
            for count in (n + 1, 16 * n + 3, 70001):
                xs = [rng.integers(0, 256, count * es, dtype=np.uint8).view(oracle.raw_dtype(dt)) for _ in range(n)]
                for shift in (0, es, 5 * es):
                    for variant, order in ((1, 0), (1, 1), (2, 0)):
                        w.tune(variant=variant, exact=True)
                        buf = [dev(x, shift) for x in xs]
                        w.all_reduce(buf, buf, count, dt, op=op, order=order)
                        torch.cuda.synchronize()
                        want = oracle.allreduce(xs, dt, op, order=order)
                        for r in range(n):
                            assert np.array_equal(back(buf[r], dt), want[r]), (n, dt, op, count, shift, variant, order, r)
            # ReduceScatter of odd blocks: every rank's own input lies at another offset; in place as well
            per = 4099
            xs = [rng.integers(0, 256, per * n * es, dtype=np.uint8).view(oracle.raw_dtype(dt)) for _ in range(n)]
            send = [dev(x) for x in xs]
            recv = [torch.zeros(per * es, dtype=torch.uint8, device="cuda") for _ in range(n)]
            w.reduce_scatter(send, recv, per, dt, op=op)
            own = [send[r][r * per * es:(r + 1) * per * es] for r in range(n)]
            w.reduce_scatter(send, own, per, dt, op=op)
            torch.cuda.synchronize()
            want = oracle.reducescatter(xs, dt, op)
            for r in range(n):
                assert np.array_equal(back(recv[r], dt), want[r]), ("rs", n, dt, op, r)
                assert np.array_equal(back(own[r].contiguous(), dt), want[r]), ("rs in place", n, dt, op, r)
    w.tune(variant=0, exact=True)
    assert all(w.status(r) == (0, 0) for r in range(n))


def scalars(dt):
    """1/8 is exact in every type; 3 overflows large values and rounds the others"""
    if dt <= L.UINT64:
        return [np.array([v & ((1 << (8 * L.DTYPE_SIZE[dt])) - 1)], dtype=oracle.raw_dtype(dt)) for v in (3, -5)]
    if dt in (L.FLOAT32, L.FLOAT64):
        return [np.array([v], dtype=np.float32 if dt == L.FLOAT32 else np.float64).view(oracle.raw_dtype(dt)) for v in (0.125, -3.3)]
    return [np.array([L.lib().hxcclHostEncode(dt, C.c_float(v))], dtype=oracle.raw_dtype(dt)) for v in (0.125, -3.0)]


@pytest.mark.parametrize("dt", [L.FLOAT32, L.FLOAT64, L.FLOAT16, L.BFLOAT16, L.FLOAT8E4M3, L.FLOAT8E5M2, L.INT64, L.INT8])
def test_one_rank_scales(dt):
    """Avg and PreMulSum over one rank against the host rules: random codes (NaN and overflow among them),
    any alignment, in place and out of place, the scalar given by value and in device memory written just
    before on the same stream."""
    import hxccl_b200 as hx
    from hxccl_b200.ops.world import World

    torch.zeros(1, device="cuda")
    comm = hx.Communicator.init_rank(hx.get_unique_id(), 1, 0)
    rng = np.random.default_rng(dt)
    es = L.DTYPE_SIZE[dt]
    with World(1, window_mb=4, wait_ms=20000) as w:
        for count in (1, 15, 128, 129, 300007):
            x = rng.integers(0, 256, count * es, dtype=np.uint8).view(oracle.raw_dtype(dt))
            for shift in (0, es):
                a, out = dev(x, shift), dev(np.zeros_like(x), shift)
                comm.all_reduce(a, out, op=hx.AVG, count=count, dtype=dt)
                torch.cuda.synchronize()
                assert np.array_equal(back(out, dt), oracle.allreduce([x], dt, L.AVG)[0]), (dt, count, shift)
                for k in scalars(dt):
                    want = oracle.allreduce([x], dt, L.SUM, scalar=k)[0]
                    b, on_device = dev(x, shift), dev(np.zeros_like(k))
                    w.all_reduce([a], [out], count, dt, scalar=k)
                    op = comm.create_premul_sum(on_device, dtype=dt, residence=L.SCALAR_DEVICE)
                    on_device.copy_(dev(k))
                    comm.all_reduce(b, b, op=op, count=count, dtype=dt)
                    torch.cuda.synchronize()
                    comm.destroy_op(op)
                    assert np.array_equal(back(out, dt), want), ("by value", dt, count, shift, k)
                    assert np.array_equal(back(b, dt), want), ("in device memory", dt, count, shift, k)
    comm.destroy()


@pytest.mark.parametrize("n", [2, 3, 8])
def test_narrow_wire_type_at_any_alignment(worlds, n):
    """hxcclAllReduceCast on fp32 buffers off the 16-byte grid, which move element by element."""
    w = worlds(n)
    w.tune(variant=0, exact=True)
    for wire, tdt in ((L.BFLOAT16, torch.bfloat16), (L.FLOAT16, torch.float16)):
        for op, count in ((L.AVG, 70001), (L.SUM, 32771)):
            g = torch.Generator().manual_seed(count + wire)
            xs = [(torch.randn(count, generator=g) * 3).float() for _ in range(n)]
            want = oracle.allreduce([x.to(tdt).view(torch.uint16).numpy().copy() for x in xs], wire, op, order=0)
            want32 = [torch.from_numpy(v.copy()).view(tdt).float().numpy() for v in want]
            for from_shift, to_shift in ((4, 4), (8, 0), (0, 12)):
                send = [dev(x.numpy(), from_shift) for x in xs]
                recv = [dev(np.zeros(count, dtype=np.float32), to_shift) for _ in range(n)]
                w.all_reduce_cast(send, recv, count, wire, op=op)
                w.all_reduce_cast(send, send, count, wire, op=op)  # in place
                torch.cuda.synchronize()
                for r in range(n):
                    for got in (recv[r], send[r]):
                        assert np.array_equal(got.cpu().numpy(), want32[r].view(np.uint8)), (n, wire, op, from_shift, to_shift, r)
    assert all(w.status(r) == (0, 0) for r in range(n))


@pytest.mark.parametrize("n,each", [(2, 20), (8, 3), (12, 5)])
def test_full_send_recv_groups(worlds, n, each):
    """Groups over all pairs of ranks: more operations than a lane takes at once (2 ranks), than the small
    parameter block holds (8 ranks: 112 lanes, 336 operations), than any launch carries (12 ranks: 1320
    operations). Sizes differ within a lane, so an operation out of order would not match its buffer."""
    w = worlds(n)
    rng = np.random.default_rng(n)
    moves = []
    for k in range(each):
        for r in range(n):
            for j in range(n):
                if r != j:
                    size = int(rng.integers(0, 6000))
                    moves.append((r, j, torch.from_numpy(rng.integers(0, 256, size + 1, dtype=np.uint8)).cuda(), size,
                                  torch.full((size + 1,), 0xEE, dtype=torch.uint8, device="cuda"), size))
    w.send_recv(moves)
    torch.cuda.synchronize()
    for r, j, src, size, dst, _ in moves:
        assert torch.equal(dst[:size], src[:size]) and int(dst[size]) == 0xEE, (n, r, j, size)
    assert all(w.status(r) == (0, 0) for r in range(n))


def test_a_world_refuses_a_capturing_stream(worlds):
    """The epochs of a world's launch are baked into its parameters, so a replay would be wrong: calls on
    a capturing stream fail, and the world works on afterwards."""
    from hxccl_b200.comm import HxcclError

    w = worlds(2)
    w.tune(variant=0, exact=True)
    x = [torch.full((50000,), float(r + 1), device="cuda") for r in range(2)]
    y = [torch.zeros_like(t) for t in x]
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        for call in (lambda: w.all_reduce(x, y, 50000, L.FLOAT32), lambda: w.all_reduce(x, y, 64, L.FLOAT32),
                     lambda: w.all_gather([t[:25000] for t in x], y, 100000),
                     lambda: w.send_recv([(0, 1, x[0], 200000, y[1], 200000)])):
            with pytest.raises(HxcclError):
                call()
        graph.capture_end()
    for count in (50000, 64):
        for t in y:
            t.zero_()
        w.all_reduce(x, y, count, L.FLOAT32)
        torch.cuda.synchronize()
        assert all(bool((t[:count] == 3).all()) for t in y)
    assert all(w.status(r) == (0, 0) for r in range(2))


def test_capture_is_refused_before_anything_is_recorded(worlds):
    """A refused call records nothing and counts nothing; what waits for nobody (transfers of a rank to
    itself, a world of one rank) is captured and replays."""
    from hxccl_b200.comm import HxcclError

    w, single = worlds(2), worlds(1)
    x = [torch.zeros(5000, device="cuda") for _ in range(2)]
    y = [torch.zeros_like(t) for t in x]
    z, marker = torch.zeros_like(x[0]), torch.zeros_like(x[0])
    nb = x[0].nbytes
    to_self, across = [(0, 0, x[0], nb, y[0], nb)], [(0, 1, x[0], nb, y[1], nb)]

    def one_rank():
        single.all_reduce([x[1]], [y[1]], 5000, L.FLOAT32)
        single.reduce_scatter([x[1]], [z], 5000, L.FLOAT32, op=L.AVG)

    one_rank()  # kernels are loaded before the capture
    torch.cuda.synchronize()
    refused, graph = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.Stream()):
        before = w.info()
        refused.capture_begin()
        marker.fill_(1)
        with pytest.raises(HxcclError):
            w.send_recv(to_self + across)
        with pytest.raises(HxcclError):
            w.all_reduce(x, y, 5000, L.FLOAT32)
        refused.capture_end()
        assert w.info() == before
        graph.capture_begin()
        w.send_recv(to_self)
        one_rank()
        graph.capture_end()
    for k in (1.0, 2.0):
        for t in x:
            t.fill_(k)
        for t in y:
            t.zero_()
        refused.replay()
        torch.cuda.synchronize()
        assert bool(marker.all()) and not any(bool(t.any()) for t in y)
        graph.replay()
        torch.cuda.synchronize()
        assert all(bool((t == k).all()) for t in (y[0], y[1], z))
    assert single.status(0) == (0, 0)


@pytest.mark.parametrize("n", [3, 6, 9, 16])
def test_orders_without_a_loop_of_their_own(worlds, n):
    """Nine ranks and more, recursive doubling over 3 and 6 ranks, binomial trees: shares of whole vectors
    per thread and shares below that, block ends inside vectors, aligned and odd buffers, in place."""
    w = worlds(n)
    rng = np.random.default_rng(100 + n)
    for dt, op in ((L.FLOAT32, L.SUM), (L.BFLOAT16, L.AVG), (L.FLOAT8E4M3, L.SUM), (L.INT32, L.AVG), (L.INT8, L.MAX)):
        es = L.DTYPE_SIZE[dt]
        for count in (2999, 300007):
            xs = [rng.integers(0, 256, count * es, dtype=np.uint8).view(oracle.raw_dtype(dt)) for _ in range(n)]
            for variant, order in ((1, 0), (1, 1), (2, 0)):
                want = oracle.allreduce(xs, dt, op, order=order)
                w.tune(variant=variant, exact=True)
                for shift in (0, es):
                    buf = [dev(x, shift) for x in xs]
                    w.all_reduce(buf, buf, count, dt, op=op, order=order)
                    torch.cuda.synchronize()
                    for r in range(n):
                        assert np.array_equal(back(buf[r], dt), want[r]), (n, dt, count, variant, order, shift, r)
            per = count // n
            send = [dev(x[:per * n], es) for x in xs]
            recv = [torch.zeros(per * es, dtype=torch.uint8, device="cuda") for _ in range(n)]
            w.reduce_scatter(send, recv, per, dt, op=op)
            out = [dev(np.zeros_like(xs[0])) if r == n - 1 else None for r in range(n)]
            w.reduce([dev(x) for x in xs], out, count, dt, n - 1, op=op)
            torch.cuda.synchronize()
            want = oracle.reducescatter([x[:per * n] for x in xs], dt, op)
            for r in range(n):
                assert np.array_equal(back(recv[r], dt), want[r]), ("rs", n, dt, count, r)
            assert np.array_equal(back(out[n - 1], dt), oracle.reduce(xs, dt, op, n - 1)), ("reduce", n, dt, count)
    w.tune(variant=0, exact=True)
    assert all(w.status(r) == (0, 0) for r in range(n))


def test_a_world_takes_the_ring_where_its_blocks_are_aligned(worlds):
    """Blocks or buffers off the 16-byte grid go to the two-shot, unless the ring is asked for."""
    n, count = 3, 3 << 17
    w = worlds(n)
    rng = np.random.default_rng(5)
    w.knob("ring_min", 1 << 20)
    try:
        for odd, shifts, forced, variant in ((0, (0, 0, 0), 0, 6), (1, (0, 0, 0), 0, 2), (2, (0, 0, 0), 0, 2), (0, (0, 4, 0), 0, 2),
                                             (1, (4, 0, 4), 6, 6)):
            w.tune(variant=forced, exact=True)
            xs = [rng.integers(0, 256, (count + odd) * 4, dtype=np.uint8).view(np.uint32) for _ in range(n)]
            send, recv = [dev(x) for x in xs], [dev(np.zeros_like(x), s) for x, s in zip(xs, shifts)]
            w.all_reduce(send, recv, count + odd, L.FLOAT32)
            torch.cuda.synchronize()
            assert w.info()["variant"] == variant, (odd, shifts, forced)
            want = oracle.allreduce(xs, L.FLOAT32, L.SUM)
            for r in range(n):
                assert np.array_equal(back(recv[r], L.FLOAT32), want[r]), (odd, shifts, forced, r)
    finally:
        w.knob("ring_min", 56 << 20)
        w.tune(variant=0, exact=True)
    assert all(w.status(r) == (0, 0) for r in range(n))


@pytest.mark.parametrize("n,kib,lines", [(7, 40, True), (7, 46, False), (8, 62, True), (12, 23, True), (12, 27, False)])
def test_lines_end_where_a_thread_would_have_two(worlds, n, kib, lines):
    """The general lines kernel (any count but 2, 4 and 8) is left before its threads take a second line."""
    w = worlds(n)
    w.tune(variant=0, exact=True)
    count = kib * 256 - 1
    rng = np.random.default_rng(n)
    xs = [rng.integers(0, 256, count * 4, dtype=np.uint8).view(np.uint32) for _ in range(n)]
    buf = [dev(x) for x in xs]
    w.all_reduce(buf, buf, count, L.FLOAT32)
    torch.cuda.synchronize()
    assert (w.info()["variant"] == 7) == lines
    want = oracle.allreduce(xs, L.FLOAT32, L.SUM)
    for r in range(n):
        assert np.array_equal(back(buf[r], L.FLOAT32), want[r]), (n, kib, r)
    assert all(w.status(r) == (0, 0) for r in range(n))
