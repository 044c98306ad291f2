"""The attention library's scratch: the same call gives the same bits whatever stream, thread, graph or context it comes from."""
import math

import pytest
import torch

from tests.gpu_util import captured_nodes, has_pre_pass

pytestmark = pytest.mark.gpu


def codes(g, *shape):
    x = torch.randn(*shape, generator=g, device="cuda").mul_(80.0).clamp_(-448, 448)
    return x.to(torch.float8_e4m3fn).view(torch.uint8)


class Decode:
    """One decode call on buffers of its own; new(seed) puts other inputs and lengths into them."""

    def __init__(self, B, Hq, Hkv, s_max, hd, seed=1):
        self.dims = (B, Hq, Hkv, hd, s_max)
        self.k, self.v = (torch.empty(B, Hkv, s_max, hd, dtype=torch.uint8, device="cuda") for _ in range(2))
        self.q = torch.empty(B, Hq, hd, dtype=torch.uint8, device="cuda")
        self.lens = torch.empty(B, dtype=torch.int32, device="cuda")
        self.sc = torch.full((3,), 1 / 80.0, device="cuda")
        self.o = torch.empty(B, Hq, hd, dtype=torch.float16, device="cuda")
        self.new(seed)

    def new(self, seed):
        B, _, _, _, s_max = self.dims
        g = torch.Generator(device="cuda").manual_seed(seed)
        for t in (self.k, self.v, self.q):
            t.copy_(codes(g, *t.shape))
        self.lens.copy_(torch.randint(s_max // 3, s_max + 1, (B,), generator=g, device="cuda"))
        torch.cuda.synchronize()

    def __call__(self, ctx, stream=None):
        B, Hq, Hkv, hd, s_max = self.dims
        stream = torch.cuda.current_stream() if stream is None else stream
        s = self.sc.data_ptr()
        ctx.Decode(self.q.data_ptr(), self.k.data_ptr(), self.v.data_ptr(), self.o.data_ptr(), 0, self.lens.data_ptr(), B, Hq, Hkv, hd, s_max, 0,
                   1.0 / math.sqrt(hd), 1.0, s, s + 4, s + 8, stream.cuda_stream)

    def result(self, ctx, stream=None):
        self.o.fill_(float("nan"))
        torch.cuda.synchronize()
        self(ctx, stream)
        torch.cuda.synchronize()
        ctx.DeviceStatus()
        assert torch.isfinite(self.o).all()
        return self.o.clone()


class Forward:
    def __init__(self, bh, s, hd, causal=1, seed=1):
        self.dims = (bh, s, hd, causal)
        self.q, self.k, self.v = (torch.empty(bh, s, hd, dtype=torch.uint8, device="cuda") for _ in range(3))
        self.sc = torch.full((3,), 1 / 80.0, device="cuda")
        self.o = torch.empty(bh, s, hd, dtype=torch.float16, device="cuda")
        self.new(seed)

    def new(self, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        for t in (self.q, self.k, self.v):
            t.copy_(codes(g, *t.shape))
        torch.cuda.synchronize()

    def __call__(self, ctx, stream=None):
        bh, s, hd, causal = self.dims
        stream = torch.cuda.current_stream() if stream is None else stream
        p = self.sc.data_ptr()
        ctx.ForwardEx(self.q.data_ptr(), self.k.data_ptr(), self.v.data_ptr(), self.o.data_ptr(), 0, bh, s, hd, causal, 0, 1.0 / math.sqrt(hd), 1.0,
                      p, p + 4, p + 8, stream.cuda_stream)

    result = Decode.result


# every plan of the decode kernel: fixed splits (cut and uncut pairs), a CTA per pair, the freely cut line
CALLS = {"splits": lambda: Decode(1, 8, 8, 1000, 128), "one split": lambda: Decode(12, 32, 32, 300, 64), "a CTA a pair": lambda: Decode(25, 32, 32, 500, 128),
         "a CTA a pair, hd 64": lambda: Decode(23, 30, 30, 900, 64), "line": lambda: Decode(5, 32, 8, 700, 128), "wide line": lambda: Decode(3, 24, 2, 900, 64),
         "forward": lambda: Forward(8, 700, 128), "forward, hd 64": lambda: Forward(3, 300, 64, 0),
         # V converted ahead, with scratch and flags
         "ahead, few tiles": lambda: Forward(4, 1300, 128, 0), "ahead, hd 64": lambda: Forward(6, 2700, 64, 0), "ahead, causal": lambda: Forward(9, 2700, 128)}
# splits that meet in a cluster: runs of one and of two or three splits, several sequences
CLUSTERS = {"cluster": lambda: Decode(1, 32, 32, 1064, 128), "cluster, runs": lambda: Decode(1, 16, 16, 2368, 128), "cluster, hd 64": lambda: Decode(5, 16, 16, 900, 64),
            "cluster, runs, hd 64": lambda: Decode(1, 16, 16, 2368, 64)}
CALLS.update(CLUSTERS)


@pytest.mark.parametrize("name", [n for n in CALLS if "forward" in n or "ahead" in n])
def test_which_forwards_take_scratch(cuda, built_libs, fa_ctx, name):
    call = CALLS[name]()
    call.result(fa_ctx)
    assert has_pre_pass(lambda: call(fa_ctx)) == ("ahead" in name)


@pytest.mark.parametrize("name", CALLS)
def test_a_graph_gives_the_bits_of_the_eager_call(cuda, built_libs, fa_ctx, name):
    call = CALLS[name]()
    call.result(fa_ctx)
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        call(fa_ctx)
        call(fa_ctx)
    for seed in (2, 3, 2):   # replayed with other inputs and lengths in the same buffers
        call.new(seed)
        want = call.result(fa_ctx)
        for _ in range(2):
            call.o.fill_(float("nan"))
            graph.replay()
            torch.cuda.synchronize()
            fa_ctx.DeviceStatus()
            assert torch.equal(call.o, want)


@pytest.mark.parametrize("name", CALLS)
def test_twenty_streams_give_the_same_bits(cuda, built_libs, fa_ctx, name):
    call = CALLS[name]()
    want = call.result(fa_ctx)
    for stream in [torch.cuda.Stream() for _ in range(20)]:
        assert torch.equal(call.result(fa_ctx, stream), want)


@pytest.mark.parametrize("name", ["a CTA a pair", "line", "forward", "ahead, few tiles", "ahead, hd 64", "ahead, causal"])
def test_streams_that_come_and_go(cuda, built_libs, fa_ctx, name):
    # each of twenty streams calls a few times, among many calls of another, so that they take each other's places; queued
    make = CALLS[name]
    busy, calls = make(), [make() for _ in range(20)]
    want = busy.result(fa_ctx)
    for c in calls:
        c.o.fill_(float("nan"))
    torch.cuda.synchronize()
    for stream, c in zip([torch.cuda.Stream() for _ in calls], calls):
        for _ in range(3):
            c(fa_ctx, stream)
        for _ in range(70):
            busy(fa_ctx)
    torch.cuda.synchronize()
    fa_ctx.DeviceStatus()
    assert all(torch.equal(c.o, want) for c in [busy, *calls])


@pytest.mark.parametrize("name,kernels,others", [("one split", 1, 0), ("splits", 2, 4), ("a CTA a pair", 1, 0), ("line", 2, 4)])
def test_nodes_of_a_captured_decode(cuda, built_libs, fa_ctx, name, kernels, others):
    # no memset node, which would part the decode kernel from the kernel ahead; nothing but the kernel where no pair is cut, and
    # else two allocations, their two frees and the kernel that clears the words
    call = CALLS[name]()
    call.result(fa_ctx)
    types = [t for t, _, _ in captured_nodes(lambda: call(fa_ctx))]
    kernel, memset, alloc, free = 0, 2, 10, 11
    assert types.count(kernel) == kernels and types.count(memset) == 0
    assert sorted(t for t in types if t != kernel) == sorted([alloc, free] * (others // 2))


@pytest.mark.parametrize("name", CLUSTERS)
def test_a_captured_cluster_leaves_its_kernel_alone(cuda, built_libs, fa_ctx, name):
    call = CLUSTERS[name]()
    call.result(fa_ctx)
    (kind, kernel, _), = captured_nodes(lambda: call(fa_ctx))
    assert kind == 0 and "fa_decode_kernel" in kernel and kernel.split("EvN")[0].endswith("Lb1EE")


@pytest.mark.parametrize("name", CLUSTERS)
def test_clusters_on_streams_that_come_and_go(cuda, built_libs, fa_ctx, name):
    test_streams_that_come_and_go(cuda, built_libs, fa_ctx, name)


@pytest.mark.parametrize("streams", [1, 4])
def test_clusters_on_threads(cuda, built_libs, fa_ctx, streams):
    # four host threads with clusters of different sizes beside a call with scratch
    import threading
    calls = [make() for make in [*CLUSTERS.values()][:3]] + [CALLS["splits"]()]
    want = [c.result(fa_ctx) for c in calls]
    for c in calls:
        c.o.fill_(float("nan"))
    ss = [torch.cuda.Stream() for _ in range(streams)]
    torch.cuda.synchronize()
    errors = []

    def work(t):
        try:
            torch.cuda.set_device(0)
            for _ in range(200):
                calls[t](fa_ctx, ss[t % streams])
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not errors, errors
    fa_ctx.DeviceStatus()
    assert all(torch.equal(c.o, w) for c, w in zip(calls, want))


def test_buffers_that_grow_and_serve_both_entry_points(cuda, built_libs, fa_ctx):
    # large, small, large again and other plans in between, on one stream, queued without a synchronisation
    ahead = [Forward(16, 3000, 128), Forward(4, 1300, 128, 0), Forward(70, 4000, 128), Forward(6, 2700, 64, 0), Forward(9, 2700, 128)]   # the third: more than is kept
    calls = [ahead[0], Forward(1, 40, 64, 0), Decode(1, 8, 8, 1000, 128), ahead[1], Decode(25, 32, 32, 500, 128), Forward(64, 2048, 128), ahead[2],
             Decode(40, 32, 8, 900, 128), ahead[3], Forward(2, 129, 64), ahead[4], Decode(1, 16, 1, 9000, 64)]
    want = [c.result(fa_ctx) for c in calls]
    assert all(has_pre_pass(lambda: c(fa_ctx)) for c in ahead)
    stream = torch.cuda.Stream()
    for order in (range(len(calls)), reversed(range(len(calls)))):
        for c in calls:
            c.o.fill_(float("nan"))
        torch.cuda.synchronize()
        for i in order:
            calls[i](fa_ctx, stream)
        torch.cuda.synchronize()
        fa_ctx.DeviceStatus()
        assert all(torch.equal(c.o, w) for c, w in zip(calls, want))


@pytest.mark.parametrize("streams,contexts", [(4, 4), (1, 4), (1, 1), (4, 1)])
@pytest.mark.parametrize("ahead", [False, True])
def test_threads(cuda, built_libs, fa_ctx, streams, contexts, ahead):
    # four host threads, each with calls of its own: streams and contexts of their own or shared
    import threading
    from goml_b200 import fa_forward as F
    make = [lambda: Decode(1, 8, 8, 1000, 128), lambda: Forward(8, 700, 128), lambda: Decode(25, 32, 32, 200, 128), lambda: Decode(5, 32, 8, 700, 128)]
    if ahead:   # forwards that share kept scratch, flags and epoch, one of them larger than another and one beside a decode call
        make = [CALLS["ahead, few tiles"], CALLS["ahead, hd 64"], lambda: Decode(5, 32, 8, 700, 128), CALLS["ahead, causal"]]
    calls = [[make[(t + i) % 4]() for i in range(3)] for t in range(4)]
    want = [[c.result(fa_ctx) for c in cs] for cs in calls]
    ss = [torch.cuda.Stream() for _ in range(streams)]
    ctxs = [F.FACreate() for _ in range(contexts)]
    for cs in calls:
        for c in cs:
            c.o.fill_(float("nan"))
    torch.cuda.synchronize()
    errors = []

    def work(t):
        try:
            torch.cuda.set_device(0)
            for _ in range(100):
                for c in calls[t]:
                    c(ctxs[t % contexts], ss[t % streams])
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not errors, errors
    fa_ctx.DeviceStatus()
    for cs, ws in zip(calls, want):
        assert all(torch.equal(c.o, w) for c, w in zip(cs, ws))
    for c in ctxs:
        c.Destroy()


LAST_CONTEXT = '''
import sys, threading, time
import torch
from goml_b200 import fa_forward as F
from tests.gpu_util import has_pre_pass
keys, ahead = int(sys.argv[1]), sys.argv[2] == "True"
codes = lambda *s: torch.randint(0, 0x60, s, dtype=torch.uint8, device="cuda")
q, k, v = codes(64, keys, 64), codes(64, keys, 64), codes(64, keys, 64)
o = torch.empty(64, keys, 64, dtype=torch.float16, device="cuda")
call = lambda ctx, s: ctx.ForwardEx(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), 0, 64, keys, 64, 1, 0, 0.1, 0.0125, 0, 0, 0, s.cuda_stream)
x = torch.zeros(1 << 20, device="cuda")
streams = [torch.cuda.Stream() for _ in range(3)]
ctx = F.FACreate()
call(ctx, streams[0])
torch.cuda.synchronize()
ctx.DeviceStatus()
want = o.clone()
assert has_pre_pass(lambda: call(ctx, torch.cuda.current_stream())) == ahead
ctx.Destroy()
for again in range(3):
    ctx, other = F.FACreate(), F.FACreate()
    call(other, streams[1])
    o.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(800_000_000)   # some 0.4 s
    call(ctx, streams[0])
    graph = torch.cuda.CUDAGraph()
    took = []
    def work():
        torch.cuda.set_device(0)
        t = time.perf_counter()
        ctx.Destroy()
        other.Destroy()                  # the last one
        took.append(time.perf_counter() - t)
    with torch.cuda.graph(graph, stream=streams[2]):
        x.add_(1)
        th = threading.Thread(target=work)
        th.start()
        th.join()
        x.add_(1)
    assert took and took[0] < 0.2, took
    x.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2).all() and torch.equal(o, want)
print("fine")
'''


@pytest.mark.parametrize("keys,ahead", [(2048, False), (4608, True)])
def test_the_last_context_goes_while_work_is_queued_and_a_capture_is_open(cuda, built_libs, keys, ahead):
    # in a process of its own: no other context of the GPU is left
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", LAST_CONTEXT, str(keys), str(ahead)], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "fine" in r.stdout, r.stdout + r.stderr
