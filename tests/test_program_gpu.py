"""Recorded runs of matvecs that zc_end_record joins into one kernel: against the calls themselves and the oracle.

The bars: x is 21-bit fixed point per 256 elements, up to 8 x 2^-20 a step for N(0, 1), 2.2e-6 of it rms (1.1e-6 for blocks
whose largest is below 4); the recorded form has the same digits of x, so that the two differ by f32 sums; a chain of
six calls passes its differences on and gate * up adds two: 2e-5.
"""
import numpy as np
import pytest

from helpers import canary_intact, dev, out_with_canary, rel_l2, run_cpp

import zinc_b200 as zb
from zinc_b200 import synth

pytestmark = pytest.mark.gpu


class Run:
    """Matrices, vectors and calls on a stream of their own; every output is followed by canary words."""

    def __init__(self, torch, seed):
        self.torch = torch
        self.stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        self.ctx = zb.Context(0, stream=self.stream.cuda_stream)
        self.dd = zb.DmmvDispatch(self.ctx)
        self.g = np.random.default_rng(seed)
        self.raw = {}
        self.beside = None

    def pad(self, n):
        """Calls beside those of a test, each worth some 2.5 us of joining: with enough of them, a run is joined that would be better
        off as launches."""
        M, K = 1024, 4096
        if self.beside is None or len(self.beside[2]) < n:
            w = synth.torch_quant_matrix(zb.Q6_K, M, K, self.torch.device("cuda"), 3)
            self.beside = w, self.vec(K), [self.out(M) for _ in range(n)]
            self.torch.cuda.synchronize()
        w, x, outs = self.beside
        for y in outs[:n]:
            self.dd.recordDispatch(zb.Q6_K, w, x, y, M, K)

    def mat(self, t, M, K):
        raw = synth.quant_matrix(self.g, t, M, K)
        w = dev(self.torch, raw)
        self.raw[w.data_ptr()] = raw
        return w

    def vec(self, n):
        return dev(self.torch, self.g.standard_normal(n).astype(np.float32))

    def out(self, n):
        return out_with_canary(self.torch, n)

    def eager_and_recorded(self, record, outs, launches, replays=1, pads=0):
        """Outputs of the calls and of a replay of the recorded ones, from the same start; every canary must hold. `pads`: calls in front
        of the recorded ones and behind them."""
        self.pad(pads)
        start = [o.clone() for o in outs]
        self.torch.cuda.synchronize()
        record()
        self.ctx.submit_and_wait()
        eager = [o.clone() for o in outs]
        n0 = self.ctx.launch_count
        with self.torch.cuda.stream(self.stream):
            self.ctx.begin_record()
            self.pad(pads)
            record()
            self.pad(pads)
            rec = self.ctx.end_record()
        assert self.ctx.launch_count - n0 == launches
        got = None
        for _ in range(replays):
            for o, s in zip(outs, start):
                o.copy_(s)
            self.torch.cuda.synchronize()
            self.ctx.replay(rec)
            self.ctx.submit_and_wait()
            now = [o.clone() for o in outs]
            assert got is None or all(self.torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0)) for a, b in zip(got, now)), "not the same bits"
            got = now
        self.ctx.free_recording(rec)
        return eager, got


# K of one, of an odd number and of many blocks; rows that start on 16-byte boundaries (Q6_K: K % 2048 == 0) and not; row
# counts around multiples of 16 and of 128
@pytest.mark.parametrize("t,M,K", [(zb.Q4_K, 16400, 256), (zb.Q4_K, 4097, 1280), (zb.Q4_K, 913, 4096), (zb.Q4_K, 321, 12288),
                                   (zb.Q6_K, 1251, 2048), (zb.Q6_K, 209, 12288), (zb.Q6_K, 10248, 256), (zb.Q6_K, 1160, 2304),
                                   (zb.Q6_K, 136, 19 * 1024), (zb.Q6_K, 240, 12032), (zb.Q6_K, 2432, 1280)])
def test_joined_matvecs_by_shape(gpu, oracle, t, M, K):
    torch, _, _ = gpu
    r = Run(torch, M + K)
    w1, w2, x1, x2 = r.mat(t, M, K), r.mat(t, M, K), r.vec(K), r.vec(K)
    a, b = r.out(M), r.out(M)
    b[:M] = 0.5
    torch.cuda.synchronize()

    def record():
        r.dd.recordDispatch(t, w1, x1, a, M, K)
        r.dd.recordDispatch(t, w2, x2, b, M, K, acc_mode=1)
    fits = K <= 12288   # beyond, the f32 kernels
    eager, got = r.eager_and_recorded(record, [a, b], 1 if fits else 4, replays=3, pads=24)
    for y, e, w, x, add in ((got[0], eager[0], w1, x1, 0.0), (got[1], eager[1], w2, x2, 0.5)):
        assert canary_intact(y, M)
        want = oracle.dmmv_f64(r.raw[w.data_ptr()], t, M, K, x.cpu().numpy()) + add
        assert rel_l2(y[:M].cpu().numpy(), want) <= 2.3e-6
        assert rel_l2(y[:M].cpu().numpy(), e[:M].cpu().numpy()) <= 1.5e-6


# Eight tiles of an SM may have their parts under way, and three warps write rows, a call each in turn. Shapes that put 8 to 35
# tiles of two consecutive calls on an SM (148 SMs), tiles of one unit (K = 256, 512), which complete out of order, and of more.
@pytest.mark.parametrize("t,shapes", [
    (zb.Q4_K, [(10240, 1024)] * 3), (zb.Q4_K, [(40000, 512)] * 2), (zb.Q4_K, [(20480, 512)] * 2 + [(10240, 512)]),
    (zb.Q4_K, [(9480, 1024), (9472, 1024), (18960, 256), (16576, 256), (18944, 512), (18960, 768)]), (zb.Q4_K, [(16576, 256)] * 7),
    (zb.Q4_K, [(304, 12288), (21312, 256), (304, 12288), (304, 12288), (21312, 256), (4736, 1024)]),
    (zb.Q6_K, [(16640, 256)] * 5), (zb.Q6_K, [(20024, 512), (300 * 8, 2048), (9472, 1024), (11008, 2048), (9480, 1280)])])
def test_many_tiles_per_sm(gpu, t, shapes):
    torch, _, _ = gpu
    r = Run(torch, 8)
    w = {s: synth.torch_quant_matrix(t, *s, torch.device("cuda"), 11 + i) for i, s in enumerate(dict.fromkeys(shapes))}
    xs = {K: r.vec(K) for _, K in shapes}
    outs = [r.out(M) for M, _ in shapes]
    torch.cuda.synchronize()

    def record():
        for y, (M, K) in zip(outs, shapes):
            r.dd.recordDispatch(t, w[M, K], xs[K], y, M, K)
        M, K = shapes[0]
        r.dd.recordDispatch(t, w[M, K], xs[K], outs[0], M, K, acc_mode=1)
    eager, got = r.eager_and_recorded(record, outs, 1, replays=20, pads=24)
    for (M, _), e, o in zip(shapes, eager, got):
        assert canary_intact(o, M)
        assert rel_l2(o[:M].cpu().numpy(), e[:M].cpu().numpy()) <= 1.5e-6


# A layer and the next one's Q, K and V of dense models from 8B to 70B, each call reading what the ones before wrote. Down
# projections with K > 12288 stay launches of their own.
@pytest.mark.parametrize("H,q_dim,kv,F,launches", [(4096, 4096, 1024, 12288, 1), (5120, 5120, 5120, 12288, 1), (5120, 5120, 5120, 13824, 3),
                                                   (4096, 4096, 1024, 14336, 3), (8192, 8192, 1024, 28672, 3)])
def test_layers_of_dense_models(gpu, H, q_dim, kv, F, launches):
    torch, _, _ = gpu
    r = Run(torch, 9)
    dd, cuda = r.dd, torch.device("cuda")
    wq, wk, wv, wo, wg, wu = (synth.torch_quant_matrix(zb.Q4_K, M, K, cuda, 21 + i) for i, (M, K) in
                              enumerate([(q_dim, H), (kv, H), (kv, H), (H, q_dim), (F, H), (F, H)]))
    wd = synth.torch_quant_matrix(zb.Q6_K, H, F, cuda, 31)
    sizes = (q_dim, kv, kv, H, F)
    q, k, v, h, act = outs = [r.out(n) for n in sizes]
    h[:H] = r.vec(H).abs()   # the weights are positive in the mean: so are all gates

    def record():
        dd.recordDispatchMulti(zb.Q4_K, [wq, wk, wv], h, [q, k, v], [q_dim, kv, kv], H)
        dd.recordDispatch(zb.Q4_K, wo, q, h, H, q_dim, acc_mode=1)
        dd.dispatchDmmvFusedGateUpSwiglu(zb.Q4_K, wg, wu, h, act, F, H)
        if launches > 1:
            r.pad(24)
        dd.recordDispatch(zb.Q6_K, wd, act, h, H, F, acc_mode=1)
        dd.recordDispatchMulti(zb.Q4_K, [wq, wk, wv], h, [q, k, v], [q_dim, kv, kv], H)
    eager, got = r.eager_and_recorded(record, outs, launches, replays=20, pads=24)
    for name, e, o, n in zip("q k v h act".split(), eager, got, sizes):
        assert canary_intact(o, n), name
        assert bool(torch.isfinite(e[:n]).all()), name
        assert rel_l2(o[:n].cpu().numpy(), e[:n].cpu().numpy()) <= 2e-5, name


def test_joined_calls_are_ordered_by_what_they_read_and_write(gpu):
    """Every way in which a call can depend on an earlier one, in one run."""
    torch, _, _ = gpu
    r = Run(torch, 5)
    dd, H, F = r.dd, 2304, 2048
    wq, wk, wv = r.mat(zb.Q4_K, H, H), r.mat(zb.Q4_K, 300, H), r.mat(zb.Q4_K, 17, H)
    wo, wg, wu, wd, wx, wh = (r.mat(zb.Q6_K, H, H), r.mat(zb.Q4_K, F, H), r.mat(zb.Q4_K, F, H), r.mat(zb.Q6_K, H, F),
                              r.mat(zb.Q4_K, H, H), r.mat(zb.Q6_K, 1301, F))
    x, q, k, v, act, h, z = r.out(H), r.out(H), r.out(300), r.out(17), r.out(F), r.out(H), r.out(1301)
    x[:H], h[:H], z[:1301] = r.vec(H), r.vec(H), r.vec(1301)
    x2 = r.vec(H)

    def record():
        dd.recordDispatchMulti(zb.Q4_K, [wq, wk, wv], x, [q, k, v], [H, 300, 17], H)
        dd.recordDispatch(zb.Q6_K, wo, q, h, H, H, acc_mode=1)                  # reads q
        dd.dispatchDmmvFusedGateUpSwiglu(zb.Q4_K, wg, wu, h, act, F, H)         # reads h
        dd.recordDispatch(zb.Q6_K, wd, act, h, H, F, acc_mode=1)                # adds to the h that the call before reads
        dd.recordDispatch(zb.Q4_K, wx, x2, x, H, H)                             # replaces the first call's x
        dd.dispatchDmmvSigmoidAcc(zb.Q6_K, wh, x, z, q, 1301, F)                # reads the new x, and q[0]
        dd.recordDispatchMulti(zb.Q4_K, [wk, wx], x2, [k, q], [300, H], H)      # replaces k and the gate's q
    outs = [x, q, k, v, act, h, z]
    for o, n in zip(outs, (H, H, 300, 17, F, H, 1301)):
        assert canary_intact(o, n)
    eager, got = r.eager_and_recorded(record, outs, 1, replays=4, pads=24)
    for name, e, o, n in zip("x q k v act h z".split(), eager, got, (H, H, 300, 17, F, H, 1301)):
        assert canary_intact(o, n), name
        assert bool(torch.isfinite(e[:n]).all()), name
        assert rel_l2(o[:n].cpu().numpy(), e[:n].cpu().numpy()) <= 2e-5, name


def test_calls_whose_ranges_overlap(gpu):
    """Outputs that meet a part of another call's x or output: windows of one buffer, 64 floats apart."""
    torch, _, _ = gpu
    r = Run(torch, 16)
    n, K = 4608, 1024
    ws = [r.mat(zb.Q4_K, n - 64 * i, K) for i in range(4)] + [r.mat(zb.Q6_K, 4096, K)]
    x, buf, y = r.vec(K), r.out(2 * n), r.out(4096)
    buf[:2 * n] = r.vec(2 * n)

    def mv(t, w, M, x, x_at, y, y_at, acc=0):
        r.dd.recordDispatch(t, w, x, y, M, K, x_offset=4 * x_at, y_offset=4 * y_at, acc_mode=acc)

    def record():
        mv(zb.Q4_K, ws[0], n, x, 0, buf, 1088)                 # the end of the next one's x
        mv(zb.Q4_K, ws[1], n - 64, buf, 128, buf, 2 * n - 4544, 1)   # adds to most of the first one's rows
        mv(zb.Q4_K, ws[2], n - 128, x, 0, buf, 64)             # replaces that x, behind it, and more of the first one's rows
        mv(zb.Q6_K, ws[4], 4096, buf, 2 * n - K, y, 0)         # the end of the second one's rows
        mv(zb.Q4_K, ws[3], n - 192, x, 0, buf, 2 * n - 4416, 1)  # adds behind the read
    eager, got = r.eager_and_recorded(record, [buf, y], 1, replays=10, pads=24)
    for e, o, m in zip(eager, got, (2 * n, 4096)):
        assert canary_intact(o, m)
        assert bool(torch.isfinite(e[:m]).all())
        assert rel_l2(o[:m].cpu().numpy(), e[:m].cpu().numpy()) <= 6e-6


def test_a_long_chain_of_calls(gpu):
    """Each call reads what the one before wrote, three buffers in turn, and every third is also read two calls later."""
    torch, _, _ = gpu
    r = Run(torch, 17)
    n = 2048
    ws, v, z = [r.mat(zb.Q6_K, n, n) for _ in range(3)], [r.out(n) for _ in range(3)], r.out(n)
    v[0][:n] = r.vec(n)

    def record():
        for i in range(9):
            r.dd.recordDispatch(zb.Q6_K, ws[i % 3], v[i % 3], v[(i + 1) % 3], n, n)
            if i % 3 == 2:
                r.dd.recordDispatch(zb.Q6_K, ws[1], v[1], z, n, n, acc_mode=1)
    outs = v + [z]
    eager, got = r.eager_and_recorded(record, outs, 1, replays=10, pads=32)
    for e, o in zip(eager, got):
        assert canary_intact(o, n)
        assert bool(torch.isfinite(e[:n]).all())
        # nine calls that each round x and add in another order
        assert rel_l2(o[:n].cpu().numpy(), e[:n].cpu().numpy()) <= 2e-5


def test_two_recordings_on_two_streams(gpu):
    """Kernels that each want all SMs, launched on two streams without a wait in between."""
    torch, _, _ = gpu
    runs = [Run(torch, 18), Run(torch, 19)]
    M, K, jobs = 20480, 1024, []
    for r in runs:
        w, x, outs = r.mat(zb.Q4_K, M, K), r.vec(K), [r.out(M) for _ in range(8)]
        torch.cuda.synchronize()

        def record(r=r, w=w, x=x, outs=outs):
            for y in outs:
                r.dd.recordDispatch(zb.Q4_K, w, x, y, M, K, acc_mode=1)
            r.pad(24)
        record()
        r.ctx.submit_and_wait()
        n0 = r.ctx.launch_count
        r.ctx.begin_record()
        record()
        jobs.append((r, outs, outs[0].clone(), r.ctx.end_record()))
        assert r.ctx.launch_count - n0 == 1
    torch.cuda.synchronize()
    for _ in range(100):
        for r, _, _, rec in jobs:
            r.ctx.replay(rec)
    for r, outs, one, rec in jobs:
        r.ctx.submit_and_wait()
        for y in outs:   # 101 additions of equal terms
            assert canary_intact(y, M)
            assert rel_l2(y[:M].cpu().numpy(), 101 * one[:M].double().cpu().numpy()) <= 101 * 2.0 ** -24 + 2e-6
        r.ctx.free_recording(rec)


def test_calls_that_are_not_joined(gpu):
    """Work of others between two calls, small matrices, and calls that write what the same run reads ahead."""
    torch, _, _ = gpu
    r = Run(torch, 6)
    M, K = 4096, 1024
    w1, w2, small = r.mat(zb.Q4_K, M, K), r.mat(zb.Q4_K, M, K), r.mat(zb.Q4_K, 64, K)
    x, a, b, c = r.vec(K), r.out(M), r.out(M), r.out(64)

    def between():
        r.dd.recordDispatch(zb.Q4_K, w1, x, a, M, K)
        with torch.cuda.stream(r.stream):
            a[:M].mul_(2.0)
        r.dd.recordDispatch(zb.Q4_K, w2, a, b, M, K)
    eager, got = r.eager_and_recorded(between, [a, b], 2)
    for e, o in zip(eager, got):
        assert torch.equal(e[:M], o[:M])

    def three():
        r.dd.recordDispatch(zb.Q4_K, small, x, c, 64, K)
        r.dd.recordDispatch(zb.Q4_K, w1, x, a, M, K)
        r.dd.recordDispatch(zb.Q4_K, w2, x, b, M, K)
    eager, got = r.eager_and_recorded(three, [a, b, c], 3, pads=24)   # what is in front, the small one, the rest
    assert torch.equal(eager[2][:64], got[2][:64])
    assert rel_l2(got[1][:M].cpu().numpy(), eager[1][:M].cpu().numpy()) <= 1.5e-6

    # the second call writes into the first one's weights (a view of them as f32)
    target = w1.view(torch.float32)[:M]
    keep = w1.clone()

    def overwrites():
        r.dd.recordDispatch(zb.Q4_K, w1, x, a, M, K)
        r.dd.recordDispatch(zb.Q4_K, w2, x, target, M, K)
    n0 = r.ctx.launch_count
    r.ctx.begin_record()
    overwrites()
    r.pad(24)
    rec = r.ctx.end_record()
    assert r.ctx.launch_count - n0 == 2
    r.ctx.replay(rec)
    r.ctx.submit_and_wait()
    got = a[:M].clone()
    w1.copy_(keep)
    torch.cuda.synchronize()
    r.dd.recordDispatch(zb.Q4_K, w1, x, a, M, K)
    r.ctx.submit_and_wait()
    assert torch.equal(got, a[:M])
    r.ctx.free_recording(rec)


def test_the_limit_for_peers_and_hand_offs_is_not_theirs(gpu):
    """A limit of one poll (zc_set_wait_limit), under which joined calls could not wait for one another."""
    torch, _, _ = gpu
    r = Run(torch, 13)
    n = 4096
    w, x, h, y = r.mat(zb.Q4_K, n, n), r.vec(n), r.out(n), r.out(n)
    r.ctx.set_wait_limit(1)

    def record():
        r.dd.recordDispatch(zb.Q4_K, w, x, h, n, n)
        r.dd.recordDispatch(zb.Q4_K, w, h, y, n, n)
    eager, got = r.eager_and_recorded(record, [h, y], 1, replays=3, pads=24)
    assert rel_l2(got[1][:n].cpu().numpy(), eager[1][:n].cpu().numpy()) <= 4e-6


def test_a_recording_ends_without_waiting(gpu):
    """Work under way on the context's own stream, which the calls are recorded from."""
    torch, _, _ = gpu
    r = Run(torch, 15)
    M, K = 4096, 1024
    w, x, outs = r.mat(zb.Q4_K, M, K), r.vec(K), [r.out(M) for _ in range(12)]
    ctx = zb.Context(0)
    dd, own = zb.DmmvDispatch(ctx), torch.cuda.ExternalStream(ctx.stream)

    def record():
        ctx.begin_record()
        for y in outs:
            dd.recordDispatch(zb.Q4_K, w, x, y, M, K)
        return ctx.end_record()
    ctx.free_recording(record())   # the kernel is loaded
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(own):
        torch.cuda._sleep(2_000_000_000)   # a second
        done.record()
    rec = record()
    assert not done.query()
    ctx.replay(rec)
    ctx.submit_and_wait()
    assert bool(outs[1][:M].any()) and torch.equal(outs[0][:M], outs[1][:M])
    ctx.free_recording(rec)
    ctx.close()


def test_calls_into_another_capture_are_its_own(gpu):
    """Between zc_begin_record and zc_end_record the caller goes to another stream, which a graph of the caller's captures."""
    torch, _, _ = gpu
    r = Run(torch, 12)
    M, K = 4096, 1024
    w1, w2, x = r.mat(zb.Q4_K, M, K), r.mat(zb.Q4_K, M, K), r.vec(K)
    outs = [r.out(M) for _ in range(4)]
    ref = [r.out(M) for _ in range(2)]
    torch.cuda.synchronize()
    r.pad(24)
    for w, y in zip((w1, w2), ref):
        r.dd.recordDispatch(zb.Q4_K, w, x, y, M, K)
    r.ctx.submit_and_wait()
    other, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    n0 = r.ctx.launch_count
    with torch.cuda.graph(graph, stream=other, capture_error_mode="relaxed"):
        r.ctx.set_stream(r.stream.cuda_stream)
        r.ctx.begin_record()
        r.ctx.set_stream(other.cuda_stream)
        for w, y in zip((w1, w2), outs[2:]):
            r.dd.recordDispatch(zb.Q4_K, w, x, y, M, K)
        r.ctx.set_stream(r.stream.cuda_stream)
        for w, y in zip((w1, w2), outs):
            r.dd.recordDispatch(zb.Q4_K, w, x, y, M, K)
        r.pad(24)
    rec = r.ctx.end_record()
    assert r.ctx.launch_count - n0 == 3   # the graph's two, and the joined ones
    r.ctx.replay(rec)
    r.ctx.submit_and_wait()
    assert not any(bool(o[:M].any()) for o in outs[2:])
    graph.replay()
    torch.cuda.synchronize()
    for i in range(2):
        assert torch.equal(outs[2 + i][:M], ref[i][:M])
        assert rel_l2(outs[i][:M].cpu().numpy(), ref[i][:M].cpu().numpy()) <= 1.5e-6
    r.ctx.free_recording(rec)


def test_a_long_run_is_several_kernels(gpu):
    """More calls than one kernel's parameters hold; each adds to the vector that the one before has written."""
    torch, _, _ = gpu
    r = Run(torch, 7)
    M, K, n = 1024, 4096, 450
    w, x, h, one = r.mat(zb.Q4_K, M, K), r.vec(K), r.out(M), r.out(M)

    def record():
        for _ in range(n):
            r.dd.recordDispatch(zb.Q4_K, w, x, h, M, K, acc_mode=1)
    r.dd.recordDispatch(zb.Q4_K, w, x, one, M, K)
    _, got = r.eager_and_recorded(record, [h], 3, replays=2, pads=24)
    # n additions of equal terms: at most n roundings of 2^-24, half of that on average
    assert rel_l2(got[0][:M].cpu().numpy(), n * one[:M].double().cpu().numpy()) <= n * 2.0 ** -24 + 2e-6


@pytest.mark.parametrize("shapes", [[(8200, 1024)] * 2, [(8200, 1024), (4104, 2048)], [(4096, 1024), (2400, 2048), (8200, 1024)]])
def test_a_recording_in_the_memory_of_an_earlier_one(gpu, shapes):
    """What a recording left behind (its tensor maps lie in memory that the next one gets) is not used by the next."""
    torch, _, _ = gpu
    r = Run(torch, 10)
    cuda = torch.device("cuda")
    for i in range(12):
        M, K = shapes[i % len(shapes)]
        t = (zb.Q4_K, zb.Q6_K)[i // 2 % 2]
        ws = [synth.torch_quant_matrix(t, M, K, cuda, 100 * i + n) for n in range(3)]
        x, outs = r.vec(K), [r.out(M) for _ in ws]

        def record():
            for w, y in zip(ws, outs):
                r.dd.recordDispatch(t, w, x, y, M, K)
        eager, got = r.eager_and_recorded(record, outs, 1, pads=24)
        for e, o in zip(eager, got):
            assert rel_l2(o[:M].cpu().numpy(), e[:M].cpu().numpy()) <= 1.5e-6, i


# Q6_K matvecs around the borders of their forms: 4.5 tiles of 16 rows per SM (148), K up to 8192 on 16-byte rows and 7424 else
@pytest.mark.parametrize("M,K", [(10656, 8192), (10640, 8192), (10656, 7424), (10656, 7680), (4736, 7424), (10656, 10240)])
def test_q6k_matvec_forms(gpu, oracle, M, K):
    torch, _, _ = gpu
    r = Run(torch, M + K)
    w, x, y = r.mat(zb.Q6_K, M, K), r.vec(K), r.out(M)
    torch.cuda.synchronize()
    r.dd.recordDispatch(zb.Q6_K, w, x, y, M, K)
    r.ctx.submit_and_wait()
    assert canary_intact(y, M)
    row = K // 256 * 210
    raw = r.raw[w.data_ptr()].reshape(-1)
    for lo in (0, M // 2 // 16 * 16, M - 64):
        want = oracle.dmmv_f64(raw[lo * row:(lo + 64) * row], zb.Q6_K, 64, K, x.cpu().numpy())
        assert rel_l2(y[lo:lo + 64].cpu().numpy(), want) <= 2.3e-6


def test_waits_that_run_out(gpu):
    """The kernel with limits that run out, with copies under way; each time a sound launch next."""
    run_cpp("test_program_waits")


def test_runs_that_are_faster_as_launches(gpu):
    """Calls that read one another's results, and runs of a few small ones, stay what they are; calls beside one another are joined."""
    torch, _, _ = gpu
    r = Run(torch, 20)
    n = 2048
    w, bufs = r.mat(zb.Q4_K, n, n), [r.out(n) for _ in range(9)]
    bufs[0][:n] = 1e-3

    def chain():
        for a, b in zip(bufs, bufs[1:]):
            r.dd.recordDispatch(zb.Q4_K, w, a, b, n, n)

    def beside(k):
        for b in bufs[1:1 + k]:
            r.dd.recordDispatch(zb.Q4_K, w, bufs[0], b, n, n)
    eager, got = r.eager_and_recorded(chain, bufs, 8)
    assert all(torch.equal(e[:n], o[:n]) for e, o in zip(eager, got))
    r.eager_and_recorded(lambda: beside(2), bufs, 2)
    r.eager_and_recorded(lambda: beside(8), bufs, 1)


def test_joining_that_is_refused(gpu):
    """A matrix without a tensor map, no memory, a node without its attribute: the calls stay launches."""
    run_cpp("test_joining")
