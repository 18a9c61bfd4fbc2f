"""Launches whose set-up runs beside the end of the stream's kernel in front of them (launch_after,
host_common.h): chains in which every call reads what the one before wrote, or writes what it
read, give the same bits as with a wait for the GPU behind every call -- eagerly, in a replayed
graph, beside the framework's own kernels and copies, and on two streams at once."""
import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu


def chain(ops, case, g, sync):
    """A dozen dependent calls on a few buffers, each used again and again; returns the buffers."""
    dev = g.device
    done = torch.cuda.synchronize if sync else (lambda: None)
    M, N, K = case
    a = torch.rand(M, K, device=dev, generator=g).sub_(0.5).mul_(2 * K ** -0.5).to(torch.bfloat16)
    b = [torch.rand(N, K, device=dev, generator=g).sub_(0.5).to(torch.bfloat16) for _ in range(2)]
    w = torch.rand(K, N, device=dev, generator=g).sub_(0.5).to(torch.bfloat16)
    c, x = torch.empty(M, N, device=dev, dtype=torch.bfloat16), torch.empty(M, K, device=dev, dtype=torch.bfloat16)
    q = torch.empty(1, M // 64, 64, K, device=dev, dtype=torch.bfloat16)
    o = torch.empty_like(q)
    y = torch.empty(M, K, device=dev)
    ones = torch.ones(K, device=dev)

    def calls():
        yield lambda: x.copy_(a)
        for i in range(4):
            yield lambda: ops.gemm(x, b[i & 1], out=c)             # reads what the last turn wrote
            yield lambda: ops.gemm(c, w, out=x)                    # over the operand just read
            if K in (64, 128):
                yield lambda: q.view(M, K).copy_(x)                # a copy of the framework's between
                yield lambda: ops.fa_fwd(q, q, q, causal=bool(i & 1), out=o)
                yield lambda: x.copy_(o.view(M, K))
            yield lambda: ops.rms_norm(x.float(), ones, out=y)
            yield lambda: ops.softmax(y, out=y)
            yield lambda: x.copy_(y)

    for call in calls():
        call()
        done()
    return [c, x, y] + ([o] if K in (64, 128) else [])


CASES = [(128, 128, 128), (1024, 1152, 128), (4096, 4096, 128), (2048, 2048, 512), (256, 4096, 4096)]


@pytest.mark.parametrize("case", CASES)
def test_chain_of_dependent_calls(pkg, gpu, case):
    want = chain(pkg.ops, case, torch.Generator(device=gpu).manual_seed(1), True)
    assert all(bool(torch.isfinite(t.float()).all()) for t in want)
    for _ in range(5):
        for got, ref in zip(chain(pkg.ops, case, torch.Generator(device=gpu).manual_seed(1), False), want):
            assert torch.equal(got, ref)
    assert pkg.ops.sync_status() == 0


def test_chain_in_a_graph_and_on_two_streams(pkg, gpu):
    case = (1024, 1152, 128)
    M, N, K = case
    g = torch.Generator(device=gpu).manual_seed(2)
    a = torch.rand(M, K, device=gpu, generator=g).sub_(0.5).to(torch.bfloat16)
    b = torch.rand(N, K, device=gpu, generator=g).sub_(0.5).to(torch.bfloat16)
    w = torch.rand(K, N, device=gpu, generator=g).sub_(0.5).mul_(0.05).to(torch.bfloat16)
    bufs = [(a.clone(), torch.empty(M, N, device=gpu, dtype=torch.bfloat16)) for _ in range(2)]

    def turn(x, c):
        pkg.ops.gemm(x, b, out=c)
        pkg.ops.gemm(c, w, out=x)
        q = x.view(1, M // 64, 64, K)
        pkg.ops.fa_fwd(q, q, q, out=c.view(-1)[:M * K].view(1, M // 64, 64, K))
        x.copy_(c.view(-1)[:M * K].view(M, K))

    x, c = a.clone(), torch.empty(M, N, device=gpu, dtype=torch.bfloat16)
    for _ in range(8):
        turn(x, c)
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    graphs = []
    for s, (xs, cs) in zip(streams, bufs):        # captured with a fork and a join in front
        with torch.cuda.stream(s):
            turn(xs, cs)                          # first calls on the stream, outside the capture
            xs.copy_(a)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                side = torch.cuda.Stream()
                side.wait_stream(s)
                with torch.cuda.stream(side):
                    xs.mul_(1.0)
                s.wait_stream(side)
                turn(xs, cs)
                turn(xs, cs)
            graphs.append(graph)
    torch.cuda.synchronize()
    for xs, _ in bufs:
        xs.copy_(a)
    torch.cuda.synchronize()
    for _ in range(4):
        for s, graph in zip(streams, graphs):
            with torch.cuda.stream(s):
                graph.replay()
    torch.cuda.synchronize()
    for xs, _ in bufs:
        assert torch.equal(xs, x)
    assert pkg.ops.sync_status() == 0


@pytest.mark.parametrize("rows,N", [(16, 2048), (300, 512), (4000, 1024), (2000, 4096), (148, 20000), (600, 30000)])
def test_weights_written_right_ahead_of_the_call(pkg, gpu, rows, N):
    """Every norm reads a weight vector and rows that the call ahead of it wrote; swiglu works in place."""
    g = torch.Generator(device=gpu).manual_seed(rows)
    x0 = torch.randn(rows, N, device=gpu, generator=g)
    w0 = torch.randn(N, device=gpu, generator=g).mul_(0.1).add_(1.0)

    def run(sync):
        done = torch.cuda.synchronize if sync else (lambda: None)
        x, y, w, b = x0.clone(), torch.empty_like(x0), w0.clone(), w0.clone()
        for i in range(12):
            for call in (lambda: w.add_(0.125), lambda: b.copy_(w).mul_(-0.5),
                         lambda: pkg.ops.layer_norm(x, w, b, out=y), lambda: w.copy_(y[i]),
                         lambda: pkg.ops.rms_norm(y, w, out=x), lambda: pkg.ops.swiglu(x, y, out=x),
                         lambda: pkg.ops.layer_norm(x, w0, b, out=x), lambda: w.copy_(w0),
                         lambda: pkg.ops.softmax(y, out=y)):
                call()
                done()
        return x, y

    want = run(True)
    assert all(bool(torch.isfinite(t).all()) for t in want)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(run(False), want))


@pytest.fixture(scope="module")
def early_writer(pkg, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("early") / "early_writer.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "device", "early_writer.cu")
    subprocess.run([pkg.build._nvcc(), *pkg.build.NVCC_FLAGS, "-shared", src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.launch_early_writer.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    return lib.launch_early_writer


@pytest.mark.parametrize("rows,N", [(16, 512), (16, 2048), (3000, 256), (2000, 1024), (2000, 4096), (148, 12000), (148, 20000),
                                    (600, 20000)])
def test_weights_written_late_by_a_kernel_that_lets_the_norm_in_early(pkg, gpu, early_writer, rows, N):
    """The norm's blocks start while the kernel in front still has the old weights in every SM's L1
    cache and has not written the new ones; the result is the new ones' all the same."""
    g = torch.Generator(device=gpu).manual_seed(N)
    x = torch.randn(rows, N, device=gpu, generator=g)
    old, new = (torch.randn(2 * N, device=gpu, generator=g) for _ in range(2))
    blocks = torch.cuda.get_device_properties(gpu).multi_processor_count
    data, sink, out = old.clone(), torch.empty(blocks * 256, device=gpu), torch.empty_like(x)
    w, b = data[:N], data[N:]
    norms = {"layer": lambda w, b: pkg.ops.layer_norm(x, w, b, out=out), "rms": lambda w, b: pkg.ops.rms_norm(x, w, out=out)}
    for norm in norms.values():
        want = norm(new[:N], new[N:]).clone()
        for _ in range(4):
            data.copy_(old)
            norm(w, b)                       # the old weights' lines in the caches of the norm's own path too
            torch.cuda.synchronize()
            assert early_writer(data.data_ptr(), new.data_ptr(), sink.data_ptr(), 2 * N, 40000, blocks,
                                torch.cuda.current_stream().cuda_stream) == 0
            norm(w, b)
            assert torch.equal(out, want)


FRONTS = {"attention": None, "one CTA": dict(M=128, N=256, K=131072, no_split=True, one_cta=True),
          "pair": dict(M=256, N=256, K=131072, no_split=True), "split": dict(M=128, N=128, K=262144)}


@pytest.mark.parametrize("front", FRONTS)
def test_the_launch_behind_leaves_the_sms_to_other_streams(pkg, gpu, front):
    """A long launch on at most half of the SMs, and one behind it that fills the machine: what
    another stream brings meanwhile runs on the SMs left, and does not wait for the first's end."""
    def bf16(*shape):
        return torch.zeros(*shape, device=gpu, dtype=torch.bfloat16)

    if FRONTS[front] is None:
        q = bf16(1, 1, 256 * (torch.cuda.get_device_properties(gpu).multi_processor_count // 2), 128)
        o = torch.empty_like(q)
        first = lambda s: pkg.ops.fa_fwd(q, q, q, out=o, flags=pkg.native.FA_NO_TAIL_SPLIT, stream=s)
    else:
        kw = dict(FRONTS[front])
        M, N, K = kw.pop("M"), kw.pop("N"), kw.pop("K")
        a, b, c = bf16(M, K), bf16(N, K), bf16(M, N)
        first = lambda s: pkg.ops.gemm(a, b, out=c, stream=s, **kw)
    a2, b2, c2 = bf16(4096, 512), bf16(4096, 512), bf16(4096, 4096)
    a3, b3, c3 = bf16(512, 128), bf16(512, 128), bf16(512, 512)
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    event = lambda: torch.cuda.Event(enable_timing=True)

    def times(second):
        torch.cuda.synchronize()
        start, end, side_end = event(), event(), event()
        with torch.cuda.stream(main):
            torch.cuda._sleep(1000000)               # half a millisecond: all is queued before anything runs
            start.record(main)
            first(main)
            if second:
                pkg.ops.gemm(a2, b2, out=c2, stream=main)
            end.record(main)
        side.wait_event(start)
        for _ in range(3):
            pkg.ops.gemm(a3, b3, out=c3, stream=side)
        side_end.record(side)
        torch.cuda.synchronize()
        return start.elapsed_time(end), start.elapsed_time(side_end)

    times(True)
    alone = min(times(False)[0] for _ in range(3))
    assert min(times(True)[1] for _ in range(3)) < 0.6 * alone
    assert pkg.ops.sync_status() == 0
