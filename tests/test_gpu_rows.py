"""Several activation rows in one pass over the weights (q4k_rows_tc.cu): Q4_K and Q5_K, against the float expectation in 64 bits."""
import numpy as np
import pytest

from backpack_b200 import q4k, synth
from oracle import q4k_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import backpack_b200 as bp

    c = bp.Q4KContext(0)
    c.set_option(q4k.OPT_ROWS_MIN_M, 2)   # every call of two rows and more, also those that other kernels serve by default
    yield c
    c.close()


def make(qtype, N, K, seed):
    """(raw file bytes, dequantised weights in 64 bits)"""
    if qtype == q4k.Q4_K:
        raw = synth.make_q4k_weights(N, K, seed)
        return raw, orc.dequant(raw, N, K).reshape(N, K).astype(np.float64)
    raw = synth.make_kq_weights(q4k.Q5_K, N, K, seed)
    return raw, orc.kq_dequant(orc.Q5_K, raw, N, K).reshape(N, K).astype(np.float64)


def upload(ctx, qtype, raw, N, K):
    return ctx.upload(q4k.pack_q4k(raw, N, K) if qtype == q4k.Q4_K else q4k.pack_kq(q4k.Q5_K, raw, N, K))


def close(y, x, w64, bias=None):
    """Bound: the activations carry 22 bits (2^-23 of the largest of a row), a super-block's products accumulate in
    float with truncation (16 steps of 2^-23 at most), the super-blocks in float: 3e-6 of |x| |w| summed covers all."""
    x64 = x.astype(np.float64)
    want = x64 @ w64.T + (0.0 if bias is None else bias.astype(np.float64))
    scale = np.sqrt((x64**2) @ (w64.T**2)) + np.abs(want) + 1e-30
    assert np.isfinite(y).all()
    rel = np.linalg.norm(y - want) / np.linalg.norm(want)
    assert np.abs((y - want) / scale).max() <= 6e-6 * np.sqrt(np.log2(w64.shape[1])) and rel <= 4e-6, (np.abs((y - want) / scale).max(), rel)


# every activation tile (8 .. 64), ragged rows of weights, one block to many, cut and whole tiles
SHAPES = [(5, 1, 256), (8, 300, 1024), (9, 256, 512), (16, 4099, 1024), (17, 511, 768), (24, 1000, 2560), (25, 257, 4096),
          (32, 640, 256), (33, 513, 1024), (48, 300, 1792), (49, 700, 1280), (64, 130, 4096), (64, 40000, 1024), (40, 300, 512), (65, 255, 1024),
          (80, 512, 1024), (96, 300, 2048), (97, 1030, 1280), (112, 200, 1280), (128, 777, 1024), (129, 300, 1024), (200, 600, 1024),
          (300, 520, 1024), (513, 260, 2048), (384, 9000, 1024)]


@pytest.mark.parametrize("qtype", [q4k.Q4_K, q4k.Q5_K], ids=["q4_k", "q5_k"])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_rows_kernel_matches_64_bits(ctx, qtype, M, N, K):
    import torch

    raw, w64 = make(qtype, N, K, M + N)
    x = synth.make_activations(M, K, M)
    bias = np.linspace(-2, 2, N).astype(np.float32)
    w = upload(ctx, qtype, raw, N, K)
    xd, bd = torch.from_numpy(x).cuda(), torch.from_numpy(bias).cuda()
    ctx.launch_count(reset=True)
    y = ctx.matmul(xd, w, bias=bd)
    assert ctx.launch_count() in (2, 3)       # the activations' layout, the matmul, the sum of tiles cut into many segments
    assert ctx.get_option(q4k.OPT_LAST_MATMUL_KERNEL) == q4k.KERNEL_ROWS
    y2 = ctx.matmul(xd, w, bias=bd)
    assert ctx.device_status() == 0
    close(y.cpu().numpy(), x, w64, bias)
    assert torch.equal(y, y2)                 # cut tiles are summed in a fixed order


@pytest.fixture(scope="module", params=[q4k.Q4_K, q4k.Q5_K], ids=["q4_k", "q5_k"])
def tall(ctx, request):
    """40003 x 4096: 157 row tiles, 17 super-blocks a CTA, so that each CTA ends one tile and begins another.  Expected
    values of sampled rows, among them the first and last of a tile and of the matrix."""
    N, K = 40003, 4096
    raw = (synth.make_q4k_weights(N, K, 71) if request.param == q4k.Q4_K else synth.make_kq_weights(q4k.Q5_K, N, K, 71)).reshape(N, -1)
    rows = np.unique(np.concatenate([np.arange(0, N, 256), np.arange(255, N, 256), [N - 1], np.random.default_rng(72).integers(0, N, 300)]))
    sample = np.ascontiguousarray(raw[rows]).reshape(-1)
    w64 = orc.dequant(sample, len(rows), K) if request.param == q4k.Q4_K else orc.kq_dequant(orc.Q5_K, sample, len(rows), K)
    yield upload(ctx, request.param, raw.reshape(-1), N, K), rows, w64.reshape(len(rows), K).astype(np.float64)


@pytest.mark.parametrize("M", [6, 16, 23, 32, 47, 64, 80, 96, 112, 128, 250])
def test_rows_kernel_of_many_units_a_cta(ctx, tall, M):
    """Rings that wrap, accumulators that alternate, whole tiles inside a share, tiles that two CTAs cut: each activation tile
    in both types (250 rows: two of 128).  To 48 rows the CTA that ends last adds a cut tile up (two launches), above a
    launch of its own does."""
    import torch

    w, rows, w64 = tall
    x = synth.make_activations(M, w.K, M)
    xd = torch.from_numpy(x).cuda()
    ctx.launch_count(reset=True)
    y = ctx.matmul(xd, w)
    assert ctx.get_option(q4k.OPT_LAST_MATMUL_KERNEL) == q4k.KERNEL_ROWS
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert ctx.launch_count() == (2 if M <= 48 else 3)
    y2 = ctx.matmul(xd, w)
    assert ctx.device_status() == 0
    close(y[:, torch.from_numpy(rows).cuda()].cpu().numpy(), x, w64)
    assert torch.equal(y, y2)


@pytest.mark.parametrize("M", [7, 20, 40, 64, 90])
def test_rows_kernel_range_of_activations_and_scales(ctx, M):
    """Rows from 1e-30 to 1e30 in magnitude, a zero row, one outlier beside small values; super-blocks whose d is zero, or
    tiny beside dmin, and blocks without a minimum."""
    import torch

    N, K = 300, 1024
    raw = synth.make_q4k_weights(N, K, 5).reshape(N * (K // 256), 144).copy()
    halves = raw[:, :4].view(np.float16)
    halves[0::7, 0] = 0.0                     # d = 0: constant blocks
    halves[1::7, 0] = 6e-8                    # the smallest half beside an ordinary dmin
    halves[2::7, 1] = 0.0                     # no minimum
    halves[3::7, :] = 0.0
    raw = raw.reshape(-1)
    w64 = orc.dequant(raw, N, K).reshape(N, K).astype(np.float64)
    x = synth.make_activations(M, K, 6)
    x *= (10.0 ** np.linspace(-30, 30, M)).astype(np.float32)[:, None]
    x[M // 2] = 0.0
    x[M // 3, 17] *= 1e6
    w = ctx.upload(q4k.pack_q4k(raw, N, K))
    y = ctx.matmul(torch.from_numpy(x).cuda(), w).cpu().numpy().astype(np.float64)
    assert ctx.device_status() == 0
    # The kernel splits a weight into sc*(q - 8) and a constant of its sub-block, so a weight that is small beside its
    # sub-block's largest keeps that one's absolute error: 2^-23 of the activation, 16 truncated steps of 2^-23 at most; where
    # that is more, 2^-39 of the row's largest activation, to 32 rows 2^-47 (2^-36 of a scaled value whose largest is 2^11).
    floor = 2.0**-39 if M > 32 else 2.0**-47
    wmax = np.repeat(np.abs(w64).reshape(N, K // 32, 32).max(axis=2), 32, axis=1)
    for t in range(M):  # each row by itself: they differ by 60 orders of magnitude
        x64 = x[t].astype(np.float64)
        want = w64 @ x64
        bound = 4e-6 * (wmax @ np.abs(x64)) + floor * np.abs(x64).max() * wmax.sum(axis=1) + 1e-37
        assert np.all(np.abs(y[t] - want) <= bound), (t, np.max(np.abs(y[t] - want) / bound))


@pytest.mark.parametrize("qtype", [q4k.Q4_K, q4k.Q5_K], ids=["q4_k", "q5_k"])
@pytest.mark.parametrize("M", [3, 8, 16, 24, 32])
@pytest.mark.parametrize("where,power", [("block", 20), ("block", 42), ("block", 80), ("sub", 17), ("sub", 24), ("sub", 28)])
def test_rows_kernel_small_values_beside_large_ones(ctx, qtype, M, where, power):
    """Activations 2^power below others of their row, whose weights are zero: in another super-block they keep all 22 bits
    (a super-block whose largest lies 2^4 below the row's has a scale of its own), in the same one down to 2^-24 of its
    largest: an error of 2^-36 of the scaled value, whose largest is at least 2^11, so 2^-47 * 2^28 = 2^-19 of a value at
    2^-28.  `close` allows 4e-6 = 2^-18."""
    import torch

    N, K = 300, 1024
    raw, _ = make(qtype, N, K, 51)
    blocks = raw.reshape(N, K // 256, -1).copy()
    x = synth.make_activations(M, K, 52)
    small = x.copy()
    if where == "block":
        blocks[:, 1, :4] = 0                  # d and dmin
        x[:, 256:512] *= np.float32(2.0**power)
        small[:, 256:512] = 0.0
    else:
        blocks[:, :, 4 + 1] &= 0xC0           # scale and minimum of every second sub-block
        blocks[:, :, 8 + 1] &= 0xC0
        one = (np.arange(K) // 32) % 8 == 1
        x[:, one] *= np.float32(2.0**power)
        small[:, one] = 0.0
    raw = blocks.reshape(-1)
    w64 = (orc.dequant(raw, N, K) if qtype == q4k.Q4_K else orc.kq_dequant(orc.Q5_K, raw, N, K)).reshape(N, K).astype(np.float64)
    y = ctx.matmul(torch.from_numpy(x).cuda(), upload(ctx, qtype, raw, N, K)).cpu().numpy()
    assert ctx.device_status() == 0
    assert (x.astype(np.float64) @ w64.T == small.astype(np.float64) @ w64.T).all()
    close(y, small, w64)


def test_rows_kernel_not_finite_stays_in_its_row(ctx):
    import torch

    M, N, K = 12, 300, 512
    raw, w64 = make(q4k.Q4_K, N, K, 9)
    x = synth.make_activations(M, K, 10)
    x[3, 100] = np.inf
    x[7, 5] = np.nan
    y = ctx.matmul(torch.from_numpy(x).cuda(), upload(ctx, q4k.Q4_K, raw, N, K)).cpu().numpy()
    bad = np.array([3, 7])
    good = np.setdiff1d(np.arange(M), bad)
    assert not np.isfinite(y[bad]).any()
    close(y[good], x[good], w64)


def test_rows_kernel_threshold_streams_and_capture(ctx):
    """Below the option's row count the streaming kernel runs; calls on several streams at once keep memory of their own, and
    each of them runs this kernel; a captured call replays."""
    import torch

    M, N, K = 12, 1000, 2048
    raw, w64 = make(q4k.Q4_K, N, K, 11)
    w = upload(ctx, q4k.Q4_K, raw, N, K)
    xs = [synth.make_activations(M, K, 20 + i) for i in range(10)]
    default = ctx.get_option(q4k.OPT_ROWS_MIN_M)
    try:
        ctx.set_option(q4k.OPT_ROWS_MIN_M, M + 1)
        close(ctx.matmul(torch.from_numpy(xs[0]).cuda(), w).cpu().numpy(), xs[0], w64)
        assert ctx.get_option(q4k.OPT_LAST_MATMUL_KERNEL) == q4k.KERNEL_STREAM
    finally:
        ctx.set_option(q4k.OPT_ROWS_MIN_M, default)
    xd = [torch.from_numpy(x).cuda() for x in xs]
    want = [ctx.matmul(x, w) for x in xd]
    ys = [torch.empty(M, N, device="cuda") for _ in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    for _ in range(20):
        for x, y, s in zip(xd, ys, streams):
            with torch.cuda.stream(s):
                ctx.matmul(x, w, out=y)
                assert ctx.get_option(q4k.OPT_LAST_MATMUL_KERNEL) == q4k.KERNEL_ROWS
    torch.cuda.synchronize()
    for x, y, v in zip(xs, ys, want):
        close(y.cpu().numpy(), x, w64)
        assert torch.equal(y, v)              # whichever stream a call runs on
    import backpack_b200 as bp

    c = bp.Q4KContext(0)
    c.set_option(q4k.OPT_ROWS_MIN_M, 2)
    try:
        y = torch.empty(M, N, device="cuda")
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):             # the handle's first call
            c.matmul(xd[0], w, out=y)
        assert c.get_option(q4k.OPT_LAST_MATMUL_KERNEL) == q4k.KERNEL_ROWS
        for x in (1, 2):
            xd[0].copy_(xd[x])
            g.replay()
            torch.cuda.synchronize()
            close(y.cpu().numpy(), xs[x], w64)
        assert c.device_status() == 0
        del g
    finally:
        c.close()


@pytest.fixture(scope="module")
def wide(ctx):
    """Calls long enough to overlap: a weight matrix and two activations with their results."""
    import torch

    M, N, K = 13, 28672, 4096
    w = upload(ctx, q4k.Q4_K, synth.make_q4k_weights(N, K, 61), N, K)
    xs = [torch.from_numpy(synth.make_activations(M, K, 62 + i)).cuda() for i in range(2)]
    ws = ctx.dequant(w).double()
    want = [x.double() @ ws.T for x in xs]
    return w, xs, want


def same(y, v):
    return float((y.double() - v).norm() / v.norm()) <= 4e-6


@pytest.mark.parametrize("M", [13, 90])
def test_rows_kernel_graphs_of_one_capture_stream_replay_side_by_side(ctx, M):
    """Two graphs captured on one stream (torch's capture stream) and replayed on two, beside eager calls on a third."""
    import torch

    N, K = 28672, 4096
    w = upload(ctx, q4k.Q4_K, synth.make_q4k_weights(N, K, 61), N, K)
    xs = [torch.from_numpy(synth.make_activations(M, K, 62 + i)).cuda() for i in range(3)]
    want = [ctx.matmul(x, w) for x in xs]
    ys = [torch.zeros(M, N, device="cuda") for _ in xs]
    graphs = []
    capture = torch.cuda.Stream()
    for x, y in zip(xs[:2], ys[:2]):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=capture):
            for _ in range(4):
                ctx.matmul(x, w, out=y)
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    for _ in range(10):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        for s in (streams[2], capture):
            with torch.cuda.stream(s):
                ctx.matmul(xs[2], w, out=ys[2])
    torch.cuda.synchronize()
    assert ctx.device_status() == 0
    for y, v in zip(ys, want):
        assert torch.equal(y, v)
    del graphs


def test_rows_kernel_batch_list_recorded_on_one_stream_and_called_on_another(ctx, wide):
    """A list of host-buffer matmuls is recorded when it is called again, then replayed whatever the stream, beside work of
    the stream it was recorded on."""
    import torch

    w, xs, want = wide
    M, K = xs[0].shape
    x_host = torch.empty(M, K, pin_memory=True)
    x_host.copy_(xs[0])
    y_host = torch.empty(M, w.N, pin_memory=True)
    batch = ctx.make_host_batch([(x_host.numpy(), w, y_host.numpy(), None)])
    streams = [torch.cuda.Stream() for _ in range(6)]
    ys = [torch.empty(M, w.N, device="cuda") for _ in streams]
    torch.cuda.synchronize()
    records = ctx.get_option(q4k.OPT_BATCH_RECORDS)
    for i in range(24):                       # (recorded on one of the first streams)
        for s, y in zip(streams, ys):
            with torch.cuda.stream(s):
                for _ in range(3):
                    ctx.matmul(xs[1], w, out=y)
        y_host.zero_()
        with torch.cuda.stream(streams[min(i, 23 - i) % 6]):
            ctx.matmul_host_batch(batch)
        assert same(y_host.cuda(), want[0]), i
    assert ctx.get_option(q4k.OPT_BATCH_RECORDS) == records + 1
    torch.cuda.synchronize()
    assert ctx.device_status() == 0
    for y in ys:
        assert same(y, want[1])


def test_rows_kernel_eager_call_beside_a_capture(ctx, wide):
    """An eager call while another stream is captured (in the mode that forbids allocations) neither fails nor spoils it."""
    import torch

    w, xs, want = wide
    ys = [torch.empty(xs[0].shape[0], w.N, device="cuda") for _ in xs]
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    import backpack_b200 as bp

    c = bp.Q4KContext(0)                      # nothing allocated yet
    try:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            c.matmul(xs[0], w, out=ys[0])
            with torch.cuda.stream(other):
                c.matmul(xs[1], w, out=ys[1])
        g.replay()
        torch.cuda.synchronize()
        assert same(ys[0], want[0]) and same(ys[1], want[1])
        del g
    finally:
        c.close()


def test_rows_kernel_memory_of_handles_and_graphs(wide):
    """A handle costs a few MB until a call needs more; memory of a captured call is used again once the graph is gone."""
    import torch

    import backpack_b200 as bp

    w, xs, want = wide
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    c = bp.Q4KContext(0)
    try:
        assert free0 - torch.cuda.mem_get_info()[0] <= 40 << 20   # (16 MB of working memory, 4 MB of scratch, the pool's granularity)
        y = torch.empty(xs[0].shape[0], w.N, device="cuda")
        free1 = None
        for i in range(12):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                c.matmul(xs[i % 2], w, out=y)
            g.replay()
            torch.cuda.synchronize()
            assert same(y, want[i % 2])
            g.reset()
            del g
            torch.cuda.synchronize()
            import time

            time.sleep(0.05)                  # (released on a thread of the driver's)
            if i == 3:
                free1 = torch.cuda.mem_get_info()[0]
        assert torch.cuda.mem_get_info()[0] >= free1 - (4 << 20)
    finally:
        c.close()


def test_rows_kernel_first_call_of_a_stream_beside_a_busy_default_stream():
    """The counters that elect the CTA which adds up a cut tile are cleared in the order of the calling stream: first calls
    on side streams (non-blocking, as torch makes them) while the default stream is busy, on a handle whose default stream
    has not been used.  600 units over 148 CTAs of whole shares of four: tiles are cut into two and the last CTA adds them
    (no launch of its own for the sums)."""
    import torch

    import backpack_b200 as bp

    M, N, K = 12, 38400, 1024
    c = bp.Q4KContext(0)
    c.set_option(q4k.OPT_ROWS_MIN_M, 2)
    try:
        raw = synth.make_q4k_weights(N, K, 31)
        w = c.upload(q4k.pack_q4k(raw, N, K))
        xd = [torch.from_numpy(synth.make_activations(M, K, 40 + i)).cuda() for i in range(4)]
        w64 = c.dequant(w).double()
        want = [x.double() @ w64.T for x in xd]
        del w64
        ys = [torch.empty(M, N, device="cuda") for _ in xd]
        streams = [torch.cuda.Stream() for _ in xd]
        a = torch.randn(8192, 8192, device="cuda")
        torch.cuda.synchronize()
        c.launch_count(reset=True)
        for _ in range(20):                   # tens of milliseconds of work on the default stream
            torch.mm(a, a)
        for x, y, s in zip(xd, ys, streams):
            with torch.cuda.stream(s):
                for _ in range(3):
                    c.matmul(x, w, out=y)
        torch.cuda.synchronize()
        assert c.device_status() == 0
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert c.launch_count() == 2 * 3 * len(xd)
        for y, v in zip(ys, want):
            assert float((y.double() - v).norm() / v.norm()) <= 4e-6
    finally:
        c.close()


# Shapes where the two kernels that could serve a call are at least 5 % apart, and the faster one.
ROUTES = [(4, 6144, 4608, "stream"), (5, 1024, 7936, "rows"), (5, 1024, 6144, "stream"), (8, 6144, 4608, "rows"), (8, 16384, 8192, "rows"),
          (8, 1024, 4096, "stream"), (8, 256, 28672, "rows"), (9, 256, 2304, "rows"), (9, 16384, 512, "stream"), (12, 1024, 1024, "stream"),
          (12, 4096, 1024, "stream"), (16, 16384, 1024, "rows"), (16, 8192, 2048, "rows"), (17, 16384, 1024, "rows"), (24, 64, 512, "rows"),
          (25, 64, 1024, "rows"), (32, 28672, 256, "rows"), (48, 1024, 512, "prefill"), (64, 28672, 1024, "rows"), (97, 256, 2048, "rows"),
          (128, 16384, 1024, "prefill"), (128, 28672, 4096, "rows"), (200, 10240, 1024, "prefill"), (257, 6144, 8192, "rows"),
          (512, 16384, 1024, "prefill"), (512, 28672, 8192, "rows"), (1024, 1024, 8192, "prefill"), (2048, 2048, 2048, "prefill")]


@pytest.mark.parametrize("M,N,K,kernel", ROUTES)
def test_calls_take_the_faster_kernel(M, N, K, kernel):
    import torch

    import backpack_b200 as bp

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the routes were timed on 148 SMs")
    c = bp.Q4KContext(0)
    try:
        for qtype, size in ((q4k.Q4_K, 144), (q4k.Q5_K, 176)):
            w = q4k.Q4KWeight(torch.zeros(N * (K // 256) * size, dtype=torch.uint8, device="cuda"), N, K, (K // 256) * size // 4, qtype)
            y = c.matmul(torch.ones(M, K, device="cuda"), w)
            got = {q4k.KERNEL_STREAM: "stream", q4k.KERNEL_PREFILL: "prefill", q4k.KERNEL_ROWS: "rows"}[c.get_option(q4k.OPT_LAST_MATMUL_KERNEL)]
            assert got == kernel and float(y.abs().max()) == 0.0 and c.device_status() == 0
    finally:
        c.close()
