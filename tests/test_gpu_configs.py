"""GPU: the benchmark configurations at full size (DeepSeek-V3 shape, 32 local of 256 experts)
against the oracle, plus size-independent properties.  Inputs are drawn on the GPU (the CPU
draw of 1.4 GB of weights takes minutes) and copied to the host for the oracle."""
import pytest
import torch

import util
from util import I, O

pytestmark = pytest.mark.gpu

PREFILL_BOOST = ((0, 8, 16, 24), 0.328)


@pytest.fixture(scope="module")
def ds_weights():
    return I.make_weights(I.DEEPSEEK_V3, seed=0, device="cuda")


def _inputs(T, weights, seed=0, boost=None, offset=0):
    d = I.make_tokens(I.DEEPSEEK_V3, T, seed, "cuda", boost)
    d.update(weights)
    d["local_expert_offset"] = offset
    d["routed_scaling_factor"] = 2.5
    return d


def _cpu(d):
    return {k: (v.cpu() if isinstance(v, torch.Tensor) else v) for k, v in d.items()}


def _check_against_oracle(T, weights, boost=None, seed=0, tile=0):
    from justgoal_b200 import MoELayer
    shape = I.DEEPSEEK_V3
    d = _inputs(T, weights, seed, boost)
    layer = MoELayer(shape)
    if tile:
        layer.set_token_tile(tile)
    out = layer.forward(*util.op_args(d))
    torch.cuda.synchronize()
    assert layer.status(T) == 0
    assert not tile or int(layer.layout(T).token_tile) == tile
    r = util.run_oracle(shape, _cpu(d))
    idx = layer.view(T, "topk_idx", torch.int32, (T, shape.top_k)).cpu()
    assert bool(O.routing_sets_equal(idx, r.topk_idx).all())
    rep = O.compare_output(out, r.output, util.ATOL, util.RTOL)
    assert rep["finite"] and rep["fail_frac"] == 0.0, rep
    return rep


def test_decode_t64(ds_weights):
    _check_against_oracle(64, ds_weights)


@pytest.mark.parametrize("tile", [0, 32, 64])
def test_mid_t901(ds_weights, tile):
    """Ragged counts at full size: the tile the layer picks for 901 tokens (128), and the 32- and 64-token kernel
    families forced through set_token_tile (several token tiles per expert, claimed chunks)."""
    _check_against_oracle(901, ds_weights, seed=7, tile=tile)


def test_token_tile_choice():
    """16 tokens while an expert expects about seven rows or fewer, 128 from about nine, 32 in between."""
    from justgoal_b200 import MoELayer
    layer = MoELayer(I.DEEPSEEK_V3)
    got = {T: int(layer.layout(T).token_tile) for T in (1, 64, 224, 256, 288, 320, 901, 4096)}
    assert got == {1: 16, 64: 16, 224: 16, 256: 32, 288: 32, 320: 128, 901: 128, 4096: 128}


def test_prefill_t4096_skewed(ds_weights):
    _check_against_oracle(4096, ds_weights, boost=PREFILL_BOOST)


def test_scaling_factor_doubling_is_exact(ds_weights):
    """out(2*f) == 2*out(f) bit for bit: the factor enters once, as a power-of-two multiple."""
    from justgoal_b200 import MoELayer
    d = _inputs(4096, ds_weights, 0, PREFILL_BOOST)
    layer = MoELayer(I.DEEPSEEK_V3)
    a = layer.forward(*util.op_args(d)).clone()
    d["routed_scaling_factor"] = 5.0
    b = layer.forward(*util.op_args(d))
    torch.cuda.synchronize()
    assert torch.equal((a.float() * 2).to(torch.bfloat16).view(torch.int16), b.view(torch.int16))


def _permuted(d, perm):
    d2 = dict(d)
    d2["routing_logits"] = d["routing_logits"][perm].contiguous()
    d2["hidden_states"] = d["hidden_states"].view(torch.uint8)[perm].contiguous().view(torch.float8_e4m3fn)
    d2["hidden_states_scale"] = d["hidden_states_scale"][:, perm].contiguous()
    return d2


def test_token_permutation_equivariance(ds_weights):
    """Permuting the tokens permutes the output rows.  With one token tile per expert (T=64) the
    result is bit-identical: columns of a tile do not interact and the combine order is by
    expert.  With several tiles per expert a token may move to another tile, whose K range is
    cut differently by the stream-K schedule (another fp32 summation order), so there only
    the last bf16 bit of a few elements may move."""
    from justgoal_b200 import MoELayer
    layer = MoELayer(I.DEEPSEEK_V3)
    for T, exact in ((64, True), (1000, False)):
        d = _inputs(T, ds_weights, 3)
        a = layer.forward(*util.op_args(d)).clone()
        perm = torch.randperm(T, generator=torch.Generator().manual_seed(1)).cuda()
        b = layer.forward(*util.op_args(_permuted(d, perm)))
        torch.cuda.synchronize()
        if exact:
            assert torch.equal(a[perm].view(torch.int16), b.view(torch.int16))
        else:
            differs = (a[perm].view(torch.int16) != b.view(torch.int16)).float().mean().item()
            assert differs < 2e-3, differs
            rep = O.compare_output(b, a[perm], 1e-3, 8e-3)      # one bf16 ulp = 2^-8 relative
            assert rep["fail_frac"] == 0.0, rep


def test_nonzero_expert_offset_matches_shifted_weights(ds_weights):
    """local_expert_offset = 32 with the same 32 weight tensors: only tokens routed to experts
    32..63 contribute; checked against the oracle."""
    from justgoal_b200 import MoELayer
    shape = I.DEEPSEEK_V3
    d = _inputs(256, ds_weights, 5, offset=32)
    layer = MoELayer(shape)
    out = layer.forward(*util.op_args(d))
    torch.cuda.synchronize()
    r = util.run_oracle(shape, _cpu(d))
    rep = O.compare_output(out, r.output, util.ATOL, util.RTOL)
    assert rep["fail_frac"] == 0.0, rep


def _share_check(shape, T, offset, rsf, seed):
    """One rank's share of an expert-parallel configuration (its local experts, all T tokens)."""
    from justgoal_b200 import MoELayer
    d = I.make_tokens(shape, T, seed, "cuda")
    d.update(I.make_weights(shape, seed, "cuda", offset))
    d["local_expert_offset"] = offset
    d["routed_scaling_factor"] = rsf
    layer = MoELayer(shape)
    out = layer.forward(*util.op_args(d))
    torch.cuda.synchronize()
    assert layer.status(T) == 0
    r = util.run_oracle(shape, _cpu(d))
    idx = layer.view(T, "topk_idx", torch.int32, (T, shape.top_k)).cpu()
    assert bool(O.routing_sets_equal(idx, r.topk_idx).all())
    rep = O.compare_output(out, r.output, util.ATOL, util.RTOL)
    assert rep["finite"] and rep["fail_frac"] == 0.0, rep


def test_ep_share_deepseek_128_local_experts():
    """The 2-GPU expert-parallel share of the 256-expert layer: 128 local experts, second rank."""
    _share_check(I.DEEPSEEK_V3.with_local(128), 512, 128, 2.5, seed=21)


def test_ep_share_qwen3_shape():
    """Qwen3-MoE shape (hidden 4096, intermediate 1536, 128 experts, 16 per rank, softmax top-8,
    renormalised, no groups), one rank's share of the 8-GPU configuration at its full T=2048."""
    _share_check(I.QWEN3_MOE, 2048, 48, 1.0, seed=22)


def test_sm_pair_kernels_match_the_single_sm_kernels():
    """The cta_group::2 family (B200MOE_PAIR=1: two CTAs of a cluster share every weight tile) computes the same
    arithmetic as the default single-SM family; the two MMA forms need not order their internal sums alike, so
    the outputs agree to a bf16 unit in the last place, not bit for bit.  Run in child processes because the
    switch is read once per process."""
    import os
    import subprocess
    import sys
    code = r"""
import sys, torch
sys.path.insert(0, %r); sys.path.insert(0, %r)
import util
from util import I
from justgoal_b200 import MoELayer
outs = []
for shape, T, seed in ((I.TINY_RENORM, 700, 31), (I.TINY_DS, 2000, 5)):
    d = I.make_inputs(shape, T, seed=seed)
    layer = MoELayer(shape)
    out = layer.forward(*util.op_args(util.to_cuda(d)))
    torch.cuda.synchronize()
    assert layer.status(T) == 0 and int(layer.layout(T).token_tile) == 128
    outs.append(out.cpu())
torch.save(outs, sys.argv[1])
""" % (util.ROOT, os.path.join(util.ROOT, "tests"))
    import tempfile
    res = {}
    with tempfile.TemporaryDirectory() as tmp:
        for pair in ("0", "1"):
            path = os.path.join(tmp, f"out{pair}.pt")
            env = dict(os.environ, B200MOE_PAIR=pair)
            r = subprocess.run([sys.executable, "-c", code, path], env=env, capture_output=True, text=True, timeout=600)
            assert r.returncode == 0, r.stderr[-2000:]
            res[pair] = torch.load(path)
    for a, b in zip(res["0"], res["1"]):
        a, b = a.float(), b.float()
        assert bool(((a - b).abs() <= 2.0 ** -7 * torch.maximum(a.abs(), b.abs()) + 1e-4).all())
        assert float((a != b).float().mean()) < 0.05


@pytest.mark.parametrize("T,tile", [(1, 0), (5, 0), (40, 0), (129, 0), (288, 0), (700, 16), (500, 32)])
def test_both_gemms_in_one_launch(ds_weights, T, tile):
    """Narrow tiles over weights that L2 cannot hold run both GEMMs in one kernel: few units that are all cut (1 and 5 tokens), whole
    ones behind both front ends, several token tiles per expert (forced tiles).  Against the two launches of the 128-token
    family: the sums agree to the order of fp32 additions, so an output differs by a unit in the last place of bf16 (2^-8) where a
    value between the GEMMs falls to the other side of an e4m3 rounding (a few in 10000; the 2-norm measured is a few 1e-4, with two tokens up to 6e-4).
    The same bits from a poisoned workspace, with stage times (two launches), with the combine fused and from a replayed graph."""
    import test_gpu_edges as edges
    from justgoal_b200 import MoELayer
    d = _inputs(T, ds_weights, seed=40 + T)
    args = util.op_args(d)
    layer = MoELayer(I.DEEPSEEK_V3)
    layer.set_token_tile(tile)
    assert int(layer.layout(T).token_tile) <= 32
    n = 3 if T <= 128 else 5
    assert layer.launches_per_forward(T) == n == edges._kernels_launched(lambda: layer.forward(*args))
    out = layer.forward(*args).clone()
    torch.cuda.synchronize()
    assert layer.status(T) == 0
    wide = MoELayer(I.DEEPSEEK_V3)
    wide.set_token_tile(128)
    assert wide.launches_per_forward(T) == n + 1
    ref = wide.forward(*args)
    rep = O.compare_output(out, ref, util.ATOL, util.RTOL)
    assert rep["finite"] and rep["fail_frac"] == 0.0, rep
    assert float((out.float() - ref.float()).norm()) <= 2e-3 * float(ref.float().norm())

    def same(other):
        torch.cuda.synchronize()
        assert layer.status(T) == 0
        assert torch.equal(out.view(torch.int16), other.view(torch.int16))

    layer.workspace(T).fill_(0xFF)
    same(layer.forward(*args))
    layer.profile_enable(2)
    assert layer.launches_per_forward(T) == n + 1 == edges._kernels_launched(lambda: layer.forward(*args))
    same(layer.forward(*args))
    assert all(v >= 0 for v in layer.profile_read(0).values())
    layer.profile_enable(0)
    layer.set_fused_combine(True)
    assert layer.launches_per_forward(T) == n - 1 == edges._kernels_launched(lambda: layer.forward(*args))
    layer.workspace(T).fill_(0xFF)
    for _ in range(3):
        fused = layer.forward(*args)
    same(fused)
    layer.set_fused_combine(False)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        replayed = layer.forward(*args)
    for _ in range(3):
        replayed.fill_(7.0)
        g.replay()
    same(replayed)


@pytest.mark.parametrize("T,tile", [(901, 16), (901, 32), (901, 64), (901, 128), (64, 0), (3, 0), (4096, 0)])
def test_forwards_repeat_their_bits(ds_weights, T, tile):
    """Sixty forwards of every tile family give the bits of the first: a read of a stage's scales that the stage's release does
    not wait for shows in one call of three (64-token tiles, 901 tokens, when it was there)."""
    from justgoal_b200 import MoELayer
    args = util.op_args(_inputs(T, ds_weights, seed=7))
    layer = MoELayer(I.DEEPSEEK_V3)
    layer.set_token_tile(tile)
    first = layer.forward(*args).clone()
    outs = [torch.equal(first.view(torch.int16), layer.forward(*args).view(torch.int16)) for _ in range(60)]
    assert layer.status(T) == 0 and all(outs)


@pytest.mark.parametrize("shape,tiles", [
    (I.DEEPSEEK_V3, {224: 16, 225: 32, 288: 32, 289: 128}),
    (I.DEEPSEEK_V3.with_local(64), {224: 16, 225: 128}),
    (I.QWEN3_MOE, {224: 16, 225: 32, 400: 32, 401: 128}),
    (I.QWEN3_MOE.with_local(128), {192: 16, 193: 128}),
    (I.TINY_DS, {56: 16, 57: 32, 72: 32, 73: 128}),                # its weights fit into L2
])
def test_token_tile_lines(shape, tiles):
    """Both sides of every line, and a workspace that serves every smaller call whatever tile that picks."""
    from justgoal_b200 import MoELayer
    layer = MoELayer(shape)
    assert {T: int(layer.layout(T).token_tile) for T in tiles} == tiles
    sizes = [int(layer.layout(T).total_bytes) for T in range(1, 520)]
    for bucket in (64, 128, 256, 512):
        assert max(sizes[:bucket]) == sizes[bucket - 1]


@pytest.mark.parametrize("T", [100, 224, 225, 400])
def test_qwen3_share_with_narrow_tiles(T):
    """One rank's share of the softmax-routed shape on both sides of the line between its narrow tiles, against the oracle."""
    _share_check(I.QWEN3_MOE, T, 48, 1.0, seed=20 + T)


@pytest.mark.parametrize("T", [112, 113, 145])
def test_routed_calls_take_the_tile_of_their_rows(ds_weights, T):
    """A routed call's experts see about twice the rows (32 of 256 experts), so it leaves the narrow tiles earlier than a forward that
    routes itself: the bits are those of the tile that its rows ask for, the launches those of a captured call."""
    import test_gpu_edges as edges
    from justgoal_b200 import MoELayer
    d = _inputs(T, ds_weights, seed=60 + T)
    layer, forced = MoELayer(I.DEEPSEEK_V3), MoELayer(I.DEEPSEEK_V3)
    tile = {112: 16, 113: 32, 145: 128}[T]
    forced.set_token_tile(tile)
    assert int(layer.layout(T).token_tile) == 16
    idx, w = layer.route(d["routing_logits"], d["routing_bias"], 2.5)
    args = (idx, w, d["hidden_states"], d["hidden_states_scale"], *[d[n] for n in (
        "gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")], 0)
    layer.workspace(T).fill_(0xFF)
    got, want = layer.forward_routed(*args).clone(), forced.forward_routed(*args)
    torch.cuda.synchronize()
    assert layer.status(T) == 0 and torch.equal(got, want)
    assert layer.launches_routed(T) == edges._kernels_launched(lambda: layer.forward_routed(*args)) == (3 if T <= 128 else 6 if tile == 128 else 5)
    layer.profile_enable(1)
    assert layer.launches_routed(T) == edges._kernels_launched(lambda: layer.forward_routed(*args)) == (4 if T <= 128 else 6)
    assert layer.launches_routed_slots(8) == 6
    layer.profile_enable(0)
    assert layer.launches_routed_slots(8) == 5


@pytest.mark.parametrize("experts", [1, 2, 3, 4, 5, 6, 8, 9])
def test_few_units_in_one_launch(ds_weights, experts):
    """16 to 144 units of GEMM1 for 148 CTAs: cut into equal pieces up to a third as many units as CTAs that start at once, dealt out
    as ranges that may end one unit and start the next up to 5/8 of all (three to five experts), whole above.  Against the two launches of the 128-token family,
    and the same bits twenty times on a poisoned workspace."""
    from justgoal_b200 import MoELayer
    T, K, E = 6, 8, I.DEEPSEEK_V3.num_experts
    d = _inputs(T, ds_weights, seed=80)
    idx = torch.arange(E - K, E, dtype=torch.int32).repeat(T, 1)                  # not on this rank
    for t in range(T):
        mine = [(t + k) % experts for k in range(min(K, experts))]
        idx[t, :len(mine)] = torch.tensor(mine, dtype=torch.int32)
    w = torch.rand(T, K, generator=torch.Generator().manual_seed(3)) + 0.1
    args = (idx.cuda(), w.cuda(), d["hidden_states"], d["hidden_states_scale"], *[d[n] for n in (
        "gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")], 0)
    layer, wide = MoELayer(I.DEEPSEEK_V3), MoELayer(I.DEEPSEEK_V3)
    wide.set_token_tile(128)
    ref = wide.forward_routed(*args)
    layer.workspace(T).fill_(0xFF)
    first = layer.forward_routed(*args).clone()
    assert int(layer.view(T, "status", torch.int32, (8,))[4]) == experts
    assert float((first - ref).norm()) <= 2e-3 * float(ref.norm())
    for k in range(20):
        if k % 5 == 0:
            layer.workspace(T).fill_(0xFF)
        assert torch.equal(first, layer.forward_routed(*args))
    assert layer.status(T) == 0 and wide.status(T) == 0


@pytest.mark.parametrize("T", [8, 30, 128])
def test_routed_calls_of_one_handle_on_two_streams(ds_weights, T):
    """Routed calls of up to 128 tokens share nothing but the handle: on two streams, a workspace each (full of other bytes), they give
    the bits that the same calls give one after the other."""
    import ctypes as C
    from justgoal_b200 import MoELayer, _lib
    layer = MoELayer(I.DEEPSEEK_V3)
    n = int(layer.layout(T).total_bytes)
    sides = []
    for k in range(2):
        d = _inputs(T, ds_weights, seed=90 + 2 * T + k)
        idx, w = layer.route(d["routing_logits"], d["routing_bias"], 2.5)
        sides.append((torch.cuda.Stream(), torch.full((n,), 0xFF, dtype=torch.uint8, device="cuda"),
                      (idx, w, d["hidden_states"], d["hidden_states_scale"],
                       *[d[m] for m in ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")])))

    def call(side, out):
        st, ws, tensors = side
        rc = _lib.lib.b200moe_forward_routed(layer._h, *[C.c_void_p(t.data_ptr()) for t in tensors], T, 0, C.c_void_p(out.data_ptr()), 0,
                                             C.c_void_p(ws.data_ptr()), n, C.c_void_p(st.cuda_stream))
        _lib.check(rc, "b200moe_forward_routed")

    want = [torch.empty(T, I.DEEPSEEK_V3.hidden, device="cuda") for _ in sides]
    torch.cuda.synchronize()
    for side, out in zip(sides, want):
        call(side, out)
        torch.cuda.synchronize()
    outs = [[torch.full_like(want[0], 7.0) for _ in range(40)] for _ in sides]
    torch.cuda.synchronize()
    for k in range(40):
        for side, o in zip(sides, outs):
            call(side, o[k])
    torch.cuda.synchronize()
    for (st, ws, _), o, ref in zip(sides, outs, want):
        assert int(ws[:4].view(torch.int32)[0]) == 0 and bool(torch.isfinite(ref).all())
        assert all(torch.equal(x, ref) for x in o)


@pytest.mark.parametrize("T", [1, 40, 128])
def test_one_fused_launch_without_rows(ds_weights, T):
    """Both GEMMs and the combine in one launch where no token has an expert on this rank: nothing in it waits for rows, and the next
    call, which has some, still finds the front end's count at zero.  Queued in turn without a host wait, also from a graph."""
    from justgoal_b200 import MoELayer
    d = _inputs(T, ds_weights, seed=50 + T)
    args = util.op_args(d)
    none = list(args)
    none[1] = args[1].clone()
    none[1][:I.DEEPSEEK_V3.num_local_experts] = -100.0            # the selection bias of the local experts: never chosen
    layer = MoELayer(I.DEEPSEEK_V3)
    want = layer.forward(*args).clone()
    layer.set_fused_combine(True)
    assert layer.launches_per_forward(T) == 2

    def turns():
        return [(layer.forward(*none), layer.forward(*none), layer.forward(*args)) for _ in range(10)]

    def check(outs):
        torch.cuda.synchronize()
        assert layer.status(T) == 0
        for a, b, c in outs:
            assert float(a.float().abs().max()) == float(b.float().abs().max()) == 0.0
            assert torch.equal(c.view(torch.int16), want.view(torch.int16))

    layer.workspace(T).fill_(0xFF)
    check(turns())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        outs = turns()
    for _ in range(3):
        for o in outs:
            for x in o:
                x.fill_(7.0)
        g.replay()
    check(outs)


@pytest.mark.parametrize("T", [40, 200])
def test_time_lines_of_one_launch_and_of_its_parts(ds_weights, T):
    """Entry and exit of GEMM1's and GEMM2's time lines: the same where one launch does both, each launch's own where stage times split it
    (GEMM2's CTAs enter after GEMM1's)."""
    from justgoal_b200 import MoELayer
    args = util.op_args(_inputs(T, ds_weights, seed=30 + T))
    layer = MoELayer(I.DEEPSEEK_V3)
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def lines():
        layer.workspace(T).fill_(0xFF)
        layer.forward(*args)
        torch.cuda.synchronize()
        assert layer.status(T) == 0
        t = layer.view(T, "trace", torch.int64, (2, sms, 16)).cpu()
        return t[:, :, 0], t[:, :, 11]

    entry, cycles = lines()
    assert torch.equal(entry[0], entry[1]) and torch.equal(cycles[0], cycles[1]) and int(cycles.min()) > 0
    layer.profile_enable(1)
    entry, cycles = lines()
    assert int(entry.min()) > 0 and int(cycles.min()) > 0
    assert int(entry[0].min()) < int(entry[1].min()) and not torch.equal(cycles[0], cycles[1])
