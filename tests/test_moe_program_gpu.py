"""Recorded MoE decode layers that zc_end_record joins into one kernel: against the calls themselves.

The bars: the same digits (Q4_K, Q6_K) or terms (MXFP4) of x and of the activations, so that the joined form differs by the order of f32
sums: 1e-6 of the logits, as much of gate and of up, whose product is the activation, and 21 bits of it (2.2e-6 rms) again in the
down projection: 1e-5. Where x is what the layer before added to, its differences go through a layer: 1e-3, and a layer that read x too
early is off by more than half."""
import pytest

from helpers import canary_intact, out_with_canary, rel_l2, run_cpp

import zinc_b200 as zb
from zinc_b200.moe_step import MoeDecode, MoeShape

pytestmark = pytest.mark.gpu


def shape(arch, H, E, k, F, L):
    q = arch == "kquant"
    return MoeShape(hidden=H, n_experts=E, top_k=k, ffn=F, t_gate_up=zb.Q4_K if q else zb.MXFP4, t_down=zb.Q6_K if q else zb.MXFP4,
                    rule=zb.ROUTE_SOFTMAX_ALL_RENORM if q else zb.ROUTE_TOPK_THEN_SOFTMAX, shared=q, oai=not q, n_layers=L, biases=not q)


class Layers:
    def __init__(self, torch, s, seed=7, layers=None):
        self.torch, self.s = torch, s
        self.stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(self.stream):
            self.ctx = zb.Context(0, stream=self.stream.cuda_stream)
            self.dd = zb.DmmvDispatch(self.ctx)
            self.step = MoeDecode.build(torch, self.dd, s, seed=seed)
        if layers:
            self.step.layers = [self.step.layers[i % len(self.step.layers)] for i in range(layers)]
        slots = self.step.routing.numel() // 2
        self.sizes = {"hidden": s.hidden, "logits": s.n_experts, "act": slots * s.ffn, "routing": 2 * slots}
        for name, n in self.sizes.items():
            setattr(self.step, name, out_with_canary(torch, n))
        self.step.routing = self.step.routing_local = self.step.routing.view(torch.int32)

    def outs(self):
        return {n: getattr(self.step, n) for n in self.sizes}

    def reset(self, hidden):
        for n, t in self.outs().items():
            t[:self.sizes[n]] = 0
        self.step.hidden[:self.s.hidden] = hidden

    def eager_and_recorded(self, record, launches, hidden=0.25, replays=3):
        torch = self.torch
        with torch.cuda.stream(self.stream):
            self.reset(hidden)
            record()
            self.ctx.submit_and_wait()
            eager = {n: t.clone() for n, t in self.outs().items()}
            n0 = self.ctx.launch_count
            self.ctx.begin_record()
            record()
            rec = self.ctx.end_record()
            assert self.ctx.launch_count - n0 == launches
            got = None
            for _ in range(replays):
                self.reset(hidden)
                self.ctx.replay(rec)
                self.ctx.submit_and_wait()
                now = {n: t.clone() for n, t in self.outs().items()}
                assert got is None or all(torch.equal(got[n].view(torch.int32), now[n].view(torch.int32)) for n in now), "not the same bits"
                got = now
            self.ctx.free_recording(rec)
        return eager, got

    def check(self, eager, got, bar=1e-5):
        slots = self.sizes["routing"] // 2
        assert self.torch.equal(eager["routing"][:slots], got["routing"][:slots])
        for n in ("logits", "act", "hidden"):
            e, g = eager[n][:self.sizes[n]].cpu().numpy(), got[n][:self.sizes[n]].cpu().numpy()
            assert rel_l2(g, e) <= (2e-6 if n == "logits" and bar == 1e-5 else bar), n
        w = [r["routing"][slots:2 * slots].view(self.torch.float32).cpu().numpy() for r in (eager, got)]
        assert rel_l2(w[1], w[0]) <= bar
        for n, t in got.items():
            assert canary_intact(t.view(self.torch.float32), self.sizes[n]), n


# experts, slots and widths at the edges: widths of an odd number of blocks of 512, widths of 64 beyond a multiple of 128, more down rows
# than SMs have tiles for, more gate and up units than the ring holds, fewer experts than SMs and several of them to a CTA
@pytest.mark.parametrize("arch,H,E,k,F,L", [
    ("kquant", 2048, 256, 8, 512, 3), ("kquant", 1280, 96, 5, 768, 2), ("kquant", 4096, 128, 8, 1024, 2), ("kquant", 1024, 64, 4, 512, 1),
    ("mxfp4", 2880, 32, 4, 2880, 2), ("mxfp4", 1088, 16, 2, 1024, 3), ("mxfp4", 1984, 24, 3, 1472, 2), ("mxfp4", 1024, 200, 4, 2624, 1)])
def test_joined_layers_by_shape(gpu, arch, H, E, k, F, L):
    torch, _, _ = gpu
    r = Layers(torch, shape(arch, H, E, k, F, L))
    r.check(*r.eager_and_recorded(r.step.record, 1, replays=20))


@pytest.mark.parametrize("arch,H,E,k,F", [("kquant", 2048, 64, 8, 512), ("mxfp4", 1984, 24, 3, 1472)])
def test_layers_that_read_what_the_one_before_wrote(gpu, arch, H, E, k, F):
    torch, _, _ = gpu
    r = Layers(torch, shape(arch, H, E, k, F, 2))
    hidden = 0.1 * torch.randn(H, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    r.step.x = r.step.hidden
    r.check(*r.eager_and_recorded(r.step.record, 1, hidden=hidden, replays=20), bar=1e-3)


# Q6_K down matrices of the selected experts below 2 MB (1.94 and 1.61): the calls hold the activations in f32 there
@pytest.mark.parametrize("H,E,k,F", [(1024, 64, 8, 256), (768, 32, 4, 512)])
def test_layers_whose_calls_hold_f32_stay_launches(gpu, H, E, k, F):
    torch, _, _ = gpu
    r = Layers(torch, shape("kquant", H, E, k, F, 2))
    eager, got = r.eager_and_recorded(r.step.record, 6)
    r.check(eager, got)
    # 21-bit activations would be 1.7e-6 off; two orders of f32 sums 1e-7
    assert rel_l2(got["hidden"][:H].cpu().numpy(), eager["hidden"][:H].cpu().numpy()) <= 5e-7


NAN, INF = float("nan"), float("inf")


def logits_of(kind, E):
    """Router logits at the edges of a selection; what is not named is 0.5."""
    v = [0.5] * E
    named = {"all the same": {}, "two levels": {i: 1.5 for i in range(3, E, 7)}, "negative zero": {i: -0.0 if i % 2 else 0.0 for i in range(E)},
             "some NaN": {0: NAN, 5: NAN, 33: 2.0, E - 1: NAN}, "all NaN": {i: NAN for i in range(E)},
             "one infinity": {40: INF, 7: 1.0}, "two infinities": {40: INF, 7: INF}, "nearly all out": {i: -INF for i in range(E) if i not in (9, E - 2)},
             "all out": {i: -INF for i in range(E)}, "lowest": {i: -3.4028234663852886e38 for i in range(2, E)}}[kind]
    for i, x in named.items():
        v[i] = x
    return v


@pytest.mark.parametrize("kind", ["all the same", "two levels", "negative zero", "some NaN", "all NaN", "one infinity", "two infinities",
                                  "nearly all out", "all out", "lowest"])
@pytest.mark.parametrize("rule", [zb.ROUTE_SOFTMAX_ALL_RENORM, zb.ROUTE_TOPK_THEN_SOFTMAX])
@pytest.mark.parametrize("E,k", [(96, 5), (250, 8)])
def test_selections_at_the_edges(gpu, kind, rule, E, k):
    """The joined kernel's selection against the router kernel's, on logits that the biases make exactly."""
    torch, _, _ = gpu
    s = shape("kquant", 1024, E, k, 512, 1)
    s.rule = rule
    r = Layers(torch, s)
    w = r.step.layers[0]
    w.router.zero_()
    w.router_bias = torch.tensor(logits_of(kind, E), device="cuda")
    torch.cuda.synchronize()
    eager, got = r.eager_and_recorded(r.step.record, 1)
    slots = k + 1
    assert torch.equal(eager["routing"][:slots], got["routing"][:slots])
    a, b = (v["routing"][slots:2 * slots].view(torch.float32) for v in (eager, got))
    assert torch.allclose(a, b, rtol=1e-6, atol=0, equal_nan=True)  # the softmax's sum in another order
    assert torch.allclose(eager["hidden"][:1024], got["hidden"][:1024], rtol=1e-4, atol=1e-5 * eager["hidden"][:1024].abs().max().item(), equal_nan=True)


@pytest.mark.parametrize("arch,H,E,k,F", [("kquant", 1024, 64, 4, 512), ("mxfp4", 1088, 16, 2, 1024)])
@pytest.mark.parametrize("odd", [NAN, INF, -INF, 3e38])
def test_an_element_of_x_that_is_no_ordinary_number(gpu, arch, H, E, k, F, odd):
    """What the calls make of it, the joined layer makes of it."""
    torch, _, _ = gpu
    r = Layers(torch, shape(arch, H, E, k, F, 1))
    r.step.x = r.step.x.clone()
    r.step.x[77] = odd
    r.step.layers[0].router[:, 77] = 0.0 if odd == 3e38 else 1.0  # (finite: the selection does not hang on the order of a sum)
    torch.cuda.synchronize()
    eager, got = r.eager_and_recorded(r.step.record, 1)
    assert torch.equal(eager["routing"][:k], got["routing"][:k])
    # activations beyond 1e30 (an infinity among the K-quants' fixed point): whether the sums over them overflow hangs on their order
    large = eager["act"][:r.sizes["act"]].abs().nan_to_num().max().item() > 1e30
    for n in ("logits", "act") if large else ("logits", "act", "hidden"):
        e, g = eager[n][:r.sizes[n]].double(), got[n][:r.sizes[n]].double()
        ordinary = e.isfinite()
        assert torch.equal(ordinary, g.isfinite()) and torch.equal(e.isnan(), g.isnan()), n
        assert torch.equal(e[~ordinary & ~e.isnan()], g[~ordinary & ~e.isnan()]), n
        assert rel_l2(g[ordinary].cpu().numpy(), e[ordinary].cpu().numpy()) <= 1e-5, n


def test_a_long_run_is_several_kernels(gpu):
    torch, _, _ = gpu
    r = Layers(torch, shape("kquant", 1024, 64, 4, 512, 2), layers=170)   # 160 in a kernel
    r.check(*r.eager_and_recorded(r.step.record, 2))


def test_calls_that_are_not_joined(gpu):
    """Layers whose calls are not one another's, whose buffers meet, or with something in between."""
    torch, _, _ = gpu
    r = Layers(torch, shape("kquant", 1024, 64, 4, 512, 2))
    step, dd = r.step, r.dd
    act, act2 = step.act, out_with_canary(torch, 5 * 512 + 256)
    x, x2 = step.x, step.x + 1.0
    layers = step.layers

    def run(*parts):
        def record():
            for layer, a, xx, between in parts:
                step.layers, step.act, step.x = [layers[layer]], a, xx
                if between:
                    between()
                step.record()
            step.layers, step.act, step.x = layers, act, x
        return record

    r.check(*r.eager_and_recorded(run((0, act, x, None), (1, act, x, None)), 1))
    r.check(*r.eager_and_recorded(run((0, act, x, None), (1, act, x2, None)), 1))
    r.check(*r.eager_and_recorded(run((0, act, x, None), (1, act2, x, None)), 1))       # other buffers throughout
    r.check(*r.eager_and_recorded(run((0, act2[256:], x, None), (1, act2, x, None)), 2))  # activations that overlap
    spare = out_with_canary(torch, 1024)
    r.check(*r.eager_and_recorded(run((0, act, x, None), (1, act, x, lambda: dd.dispatchSwiglu(x2, x2, spare, 512))), 3))
    # selections into a place of their own in between
    other = torch.zeros_like(step.routing)

    def route_again():
        w = layers[1]
        dd.dispatchMoeRouterTopk(x2, w.router, r.step.logits, other, 64, 1024, 4, rule=r.s.rule, shared_slot=True)
    r.check(*r.eager_and_recorded(run((0, act, x, None), (1, act, x, route_again)), 3))


def test_two_recordings_on_two_streams(gpu):
    torch, _, _ = gpu
    a, b = Layers(torch, shape("kquant", 2048, 64, 8, 512, 3)), Layers(torch, shape("mxfp4", 1920, 24, 3, 1920, 3))
    recs = []
    for r in (a, b):
        with torch.cuda.stream(r.stream):
            r.reset(0.25)
            r.step.record()
            r.ctx.submit_and_wait()
            r.eager = {n: t.clone() for n, t in r.outs().items()}
            r.ctx.begin_record()
            r.step.record()
            recs.append(r.ctx.end_record())
            r.ctx.submit_and_wait()
    for _ in range(20):
        for r, rec in zip((a, b), recs):
            with torch.cuda.stream(r.stream):
                r.reset(0.25)
                r.ctx.replay(rec)
    for r, rec in zip((a, b), recs):
        r.ctx.submit_and_wait()
        r.check(r.eager, r.outs())
        r.ctx.free_recording(rec)


def test_waits_that_run_out(gpu):
    """The kernel with limits that run out, with copies under way; each time a sound launch next."""
    run_cpp("test_moe_waits")
