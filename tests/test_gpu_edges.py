"""Ragged and boundary cases of the CUDA path against the oracle: one token, the first size past the
fused small-T front end, several permutation slices, every token colliding on the same experts,
ragged last tiles.  Output tolerance as stated for the operator; integer structures exact."""
import dataclasses
import functools

import pytest
import torch

import util
from util import I, O

pytestmark = pytest.mark.gpu


def _forward(shape, d, layer=None):
    from justgoal_b200 import MoELayer
    layer = layer or MoELayer(shape)
    out = layer.forward(*util.op_args(util.to_cuda(d)))
    torch.cuda.synchronize()
    T = int(d["hidden_states"].shape[0])
    assert layer.status(T) == 0
    return layer, out


def _check_output(shape, d, out):
    want = util.run_oracle(shape, d).output
    rep = O.compare_output(out, want, util.ATOL, util.RTOL)
    assert rep["fail_frac"] == 0.0, rep


def _check_tables(shape, d, layer, T):
    """counts, segment alignment, ascending tokens inside every expert segment, padding rows = -1,
    pair_row pointing back at the pair's token."""
    r = util.run_oracle(shape, d, keep_inter=True)
    El, K = shape.num_local_experts, shape.top_k
    rows_cap = int(layer.layout(T).rows_cap)
    counts = layer.view(T, "counts", torch.int32, (El,)).cpu()
    row0 = layer.view(T, "expert_row0", torch.int32, (El + 1,)).cpu()
    row_token = layer.view(T, "row_token", torch.int32, (rows_cap,)).cpu()
    pair_row = layer.view(T, "pair_row", torch.int32, (T, K)).cpu()
    topk = layer.view(T, "topk_idx", torch.int32, (T, K)).cpu()
    want = torch.tensor([len(r.expert_tokens.get(e, [])) for e in range(El)], dtype=torch.int32)
    assert torch.equal(counts, want)
    for e in range(El):
        a, c = int(row0[e]), int(counts[e])
        assert a % 16 == 0 and int(row0[e + 1]) - a == (c + 15) // 16 * 16
        if c:
            assert torch.equal(row_token[a:a + c].long(), r.expert_tokens[e])
        assert bool((row_token[a + c:int(row0[e + 1])] == -1).all())
    off = int(d["local_expert_offset"])
    local = (topk >= off) & (topk < off + El)
    t_of_pair = torch.arange(T).unsqueeze(1).expand(T, K)
    assert torch.equal(row_token[pair_row[local].long()].long(), t_of_pair[local])


def test_single_token():
    shape = I.TINY_DS
    d = I.make_inputs(shape, 1, seed=21)
    layer, out = _forward(shape, d)
    _check_output(shape, d, out)


@pytest.mark.parametrize("tile", [0, 16, 32, 64])
@pytest.mark.parametrize("T", [128, 129, 257])
def test_around_the_fused_front_end_boundary(T, tile):
    """T = 128 is the last size of the fused permute + gather launch, 129 the first of the sliced
    permutation (two slices of 1024 pairs), 257 crosses into a third slice.  Run with the tile the layer picks
    (128 tokens here) and with every narrow kernel family forced (several token tiles per expert)."""
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS
    d = I.make_inputs(shape, T, seed=22 + T)
    layer = MoELayer(shape)
    layer.set_token_tile(tile)
    layer, out = _forward(shape, d, layer)
    _check_output(shape, d, out)
    _check_tables(shape, d, layer, T)


def test_many_slices_top4():
    """top-4 shape, 700 tokens = 2800 pairs = 3 slices; a token's pairs straddle slice borders."""
    shape = I.TINY_RENORM
    d = I.make_inputs(shape, 700, seed=31)
    layer, out = _forward(shape, d)
    _check_output(shape, d, out)
    _check_tables(shape, d, layer, 700)


def test_all_tokens_collide_on_the_same_experts():
    """Identical routing rows: every token picks the same top-k experts, so a few experts receive T
    rows each (several token tiles with a ragged last one) and all others none."""
    shape = I.TINY_DS
    T = 300
    d = I.make_inputs(shape, T, seed=41)
    d["routing_logits"] = d["routing_logits"][:1].repeat(T, 1).contiguous()
    layer, out = _forward(shape, d)
    _check_output(shape, d, out)
    _check_tables(shape, d, layer, T)
    counts = layer.view(T, "counts", torch.int32, (shape.num_local_experts,)).cpu()
    assert set(counts.tolist()) <= {0, T}


def test_small_forwards_back_to_back_without_a_host_wait():
    """Up to 128 tokens the forward is four launches and nothing else on the stream, each allowed to start under
    the tail of the one before: the front end of call n+1 overlaps the combine of call n, clears the head of the
    workspace itself, meets at two words owned by the handle, and GEMM1 schedules itself from the routing result
    while the front end still gathers.  Twelve forwards with two alternating token sets and sizes are queued with
    no host wait in between; every result must match the oracle and the error word must stay clear."""
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS
    layer = MoELayer(shape)
    cases = [I.make_inputs(shape, T, seed=seed) for T, seed in ((64, 61), (7, 62), (128, 63))]
    args = [util.op_args(util.to_cuda(d)) for d in cases]
    outs = []
    for n in range(12):
        outs.append((n % 3, layer.forward(*args[n % 3]).clone()))
    torch.cuda.synchronize()
    for T in (64, 7, 128):
        assert layer.status(T) == 0
    want = [util.run_oracle(shape, d).output for d in cases]
    for k, out in outs:
        rep = O.compare_output(out, want[k], util.ATOL, util.RTOL)
        assert rep["fail_frac"] == 0.0, (k, rep)
    # the same inputs give the same bits every time (fixed summation order, whoever was quick or slow)
    for k in range(3):
        same = [o for kk, o in outs if kk == k]
        assert all(torch.equal(same[0].view(torch.int16), o.view(torch.int16)) for o in same[1:])


@pytest.mark.parametrize("shape_name,T,tile", [("TINY_DS", 64, 16), ("TINY_DS", 150, 32), ("TINY_DS", 400, 64),
                                               ("TINY_RENORM", 20, 16), ("TINY_RENORM", 130, 32)])
def test_fused_combine_equals_the_combine_kernel_bit_for_bit(shape_name, T, tile):
    """With the fused combine switched on and narrow token tiles the forward has no combine launch: the GEMM2 unit
    that delivers a token's last row sums the token's rows in its epilogue.  forward_routed keeps the separate combine kernel; both add the same
    rows in the same order, so the bf16 outputs must be identical - including tokens without a local expert (zero
    rows) and a hidden size that is not a multiple of 256 (TINY_RENORM: the last unit has one weight tile)."""
    from justgoal_b200 import MoELayer
    shape = getattr(I, shape_name)
    d = I.make_inputs(shape, T, seed=70 + T)
    layer = MoELayer(shape)
    layer.set_token_tile(tile)                         # every narrow kernel family, whatever the layer would pick
    assert layer.launches_per_forward(T) == (4 if T <= 128 else 6)
    layer.set_fused_combine(True)                      # off by default
    assert layer.launches_per_forward(T) == (3 if T <= 128 else 5)
    _, out = _forward(shape, d, layer)
    assert int(layer.layout(T).token_tile) == tile
    _check_output(shape, d, out)
    K = shape.top_k
    idx = layer.view(T, "topk_idx", torch.int32, (T, K)).clone()
    w = layer.view(T, "topk_w", torch.float32, (T, K)).clone()
    dc = util.to_cuda(d)
    out2 = layer.forward_routed(idx, w, dc["hidden_states"], dc["hidden_states_scale"], dc["gemm1_weights"],
                                dc["gemm1_weights_scale"], dc["gemm2_weights"], dc["gemm2_weights_scale"],
                                int(d["local_expert_offset"]), out_dtype=torch.bfloat16)
    torch.cuda.synchronize()
    assert layer.status(T) == 0
    assert torch.equal(out.view(torch.int16), out2.view(torch.int16))


@pytest.mark.parametrize("counts", [(1, 31, 32, 33, 96, 97, 128, 129), (127, 160, 161, 255, 256, 257, 16, 64)])
@pytest.mark.parametrize("hidden,intermediate", [(512, 256), (1536, 1152)])
def test_part_full_128_token_tiles(counts, hidden, intermediate):
    """128-token tiles at every edge of their 32-row quarters, through the instance for mostly part-full tiles (few tokens)
    and the one for full tiles (the same tokens among many without a local expert): the oracle's result, and the same
    bits from both.  The workspace is poisoned: quarters that are left out must not matter.  (The second size has just the
    K blocks from which rows that a stage held earlier are cleared, the first one fewer.)"""
    import dataclasses
    from justgoal_b200 import MoELayer
    shape = dataclasses.replace(I.TINY_DS, hidden=hidden, intermediate=intermediate)
    few, many = max(counts), 1100                        # below / above 128 expected rows per expert
    assert few * shape.top_k / shape.num_experts < 128 <= many * shape.top_k / shape.num_experts
    d = I.make_inputs(shape, many, seed=17)
    idx = torch.full((many, shape.top_k), shape.num_experts - 1, dtype=torch.int32)       # not on this rank
    for k, n in enumerate(counts):
        idx[:n, k] = 2 * k
    w = torch.rand(many, shape.top_k, generator=torch.Generator().manual_seed(3)) + 0.1
    want, _, _ = O.run_experts(d["hidden_states"][:few], d["hidden_states_scale"][:, :few].contiguous(), d["gemm1_weights"],
                               d["gemm1_weights_scale"], d["gemm2_weights"], d["gemm2_weights_scale"], w[:few], idx[:few].long(),
                               0, shape.num_experts)
    dc = util.to_cuda(d)
    layer = MoELayer(shape)
    layer.set_token_tile(128)
    outs = []
    for T in (few, many):
        layer.workspace(T).fill_(0xFF)
        out = layer.forward_routed(idx[:T].cuda(), w[:T].cuda(), dc["hidden_states"][:T], dc["hidden_states_scale"][:, :T].contiguous(),
                                   dc["gemm1_weights"], dc["gemm1_weights_scale"], dc["gemm2_weights"], dc["gemm2_weights_scale"],
                                   0, out_dtype=torch.bfloat16)
        torch.cuda.synchronize()
        assert layer.status(T) == 0
        outs.append(out.clone())
    rep = O.compare_output(outs[0], want.to(torch.bfloat16), util.ATOL, util.RTOL)
    assert rep["finite"] and rep["fail_frac"] == 0.0, rep
    assert torch.equal(outs[0].view(torch.int16), outs[1][:few].view(torch.int16))
    assert bool((outs[1][few:].float() == 0).all())


@pytest.mark.parametrize("tma_gather", [False, True])
@pytest.mark.parametrize("hidden,intermediate", [(128, 128), (384, 640), (1152, 1024)])
def test_scale_ring_of_the_128_token_tiles(hidden, intermediate, tma_gather):
    """K blocks fewer than the scales travel ahead (1, 3, 5), just as many as the ring holds (8) and one more (9)."""
    import dataclasses
    from justgoal_b200 import MoELayer
    shape = dataclasses.replace(I.TINY_DS, hidden=hidden, intermediate=intermediate)
    d = I.make_inputs(shape, 300, seed=23)
    layer = MoELayer(shape)
    layer.set_token_tile(128)
    layer.set_tma_gather(tma_gather)
    layer.workspace(300).fill_(0xFF)
    _, out = _forward(shape, d, layer)
    _check_output(shape, d, out)


@pytest.mark.parametrize("T", [2369, 9473])
def test_combine_batches(T):
    """Token counts from which a combine CTA takes two / eight tokens at a time, with a ragged last batch."""
    shape = I.TINY_RENORM
    d = I.make_inputs(shape, T, seed=T)
    layer, out = _forward(shape, d)
    _check_output(shape, d, out)


def _pieces(units, KB, kpb, slots_per_cta, piece_cost, grid):
    """Pieces of a left-over unit, as gemm.cuh's size_chunks states the rule."""
    tail, groups = units % grid, -(-KB // kpb)
    best, length = groups * kpb, groups
    for n in range(2, 9):
        if tail * n > grid * slots_per_cta:
            break
        size = -(-groups // n)
        cost = -(-tail * n // grid) * (size * kpb + piece_cost + n)
        if cost < best:
            best, length = cost, size
    return -(-groups // length)


@functools.lru_cache(maxsize=1)
def _wide_intermediate():
    """32 K blocks in GEMM2: enough for every tile family to cut left-over units."""
    shape = dataclasses.replace(I.TINY_DS, hidden=1024, intermediate=4096, num_local_experts=8)
    return shape, I.make_inputs(shape, 1100, seed=29)


@pytest.mark.parametrize("tiles", [1, 3, 5, 7, 12, 25])
@pytest.mark.parametrize("tile,full", [(16, False), (32, False), (64, False), (128, False), (128, True)])
def test_left_over_units_cut_along_k(tile, full, tiles):
    """Claimed pieces of GEMM2 in every tile family (both instances of the 128-token tiles), GEMM1's static tails beside them on
    both sides of half a grid of left-over units, without and with whole units before (32 units of GEMM1 and 4 of GEMM2 per tile; with 12
    tiles the partial-sum slots end the search for 128-token tiles, with 25 GEMM2's units stay whole).  The oracle's result, the same bits from a second call on a
    poisoned workspace, and as many pieces as the rule says."""
    from justgoal_b200 import MoELayer, _lib
    shape, d = _wide_intermediate()
    spread = [tiles // 8 + (e < tiles % 8) for e in range(8)]
    rows = [k * tile - (3 * e + 1) % (tile - 1) if k else 0 for e, k in enumerate(spread)]
    used = max(rows)
    T = 1100 if full else used
    assert (T * shape.top_k / shape.num_experts >= 128) == full
    idx = torch.full((T, shape.top_k), shape.num_experts - 1, dtype=torch.int32)          # not on this rank
    for e, n in enumerate(rows):
        idx[:n, e] = e
    w = torch.rand(T, shape.top_k, generator=torch.Generator().manual_seed(5)) + 0.1
    x, sc = d["hidden_states"][:T], d["hidden_states_scale"][:, :T].contiguous()
    wts = [d[n] for n in ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")]
    want, _, _ = O.run_experts(x[:used], sc[:, :used].contiguous(), *wts, w[:used], idx[:used].long(), 0, shape.num_experts)
    layer = MoELayer(shape)
    layer.set_token_tile(tile)
    args = [t.cuda() for t in (idx, w, x, sc, *wts)]
    grid, outs = _lib.lib.b200moe_num_sms(), []
    for _ in range(2):
        layer.workspace(T).fill_(0xFF)
        outs.append(layer.forward_routed(*args, 0, out_dtype=torch.bfloat16).clone())
        torch.cuda.synchronize()
        assert layer.status(T) == 0
        arrived = layer.view(T, "sk_count", torch.int32, (2, 4 * grid + 4)).cpu()
        units = 4 * tiles
        want_pieces = _pieces(units, 32, 2 if tile == 16 else 1, {16: 16, 32: 8, 64: 4, 128: 2}[tile],
                              8 if tile < 128 else 12 if full else 6, grid)
        assert (want_pieces > 1) == (tiles < 25)
        first = arrived[1, :4 * (units % grid):4]                  # of the first group of warps of every left-over unit
        assert set((first & 0xFF).tolist()) == {want_pieces if want_pieces > 1 else 0}
        if tile <= 32:
            tail = 32 * tiles % grid
            assert bool((arrived[0, :4 * tail:4] > 0).all())
    rep = O.compare_output(outs[0][:used], want.to(torch.bfloat16), util.ATOL, util.RTOL)
    assert rep["finite"] and rep["fail_frac"] == 0.0, rep
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    assert bool((outs[0][used:].float() == 0).all())


@pytest.mark.parametrize("tile,T", [(16, 20), (16, 100), (32, 180), (64, 400)])
def test_fused_combine_behind_cut_units(tile, T):
    """The fused combine when GEMM2's units are cut: the warps that add a unit's pieces up deliver its rows."""
    from justgoal_b200 import MoELayer, _lib
    shape, d = _wide_intermediate()
    d = {k: v[:T] if k in ("routing_logits", "hidden_states") else v for k, v in d.items()}
    d["hidden_states_scale"] = d["hidden_states_scale"][:, :T].contiguous()
    layer = MoELayer(shape)
    layer.set_token_tile(tile)
    _, separate = _forward(shape, d, layer)
    _check_output(shape, d, separate)
    layer.set_fused_combine(True)
    for _ in range(2):
        layer.workspace(T).fill_(0xFF)
        _, fused = _forward(shape, d, layer)
        assert torch.equal(fused.view(torch.int16), separate.view(torch.int16))
        grid = _lib.lib.b200moe_num_sms()
        assert int(layer.view(T, "sk_count", torch.int32, (2, 4 * grid + 4))[1, 0]) & 0xFF > 1


def _kernel_names(fn):
    """Names of the kernel nodes of the CUDA graph that captures one call of fn, in the order of the graph's node list."""
    import ctypes as C

    class Params(C.Structure):                         # CUDA_KERNEL_NODE_PARAMS_v2
        _fields_ = [("func", C.c_void_p), ("dims", C.c_uint * 7), ("kernel_params", C.c_void_p), ("extra", C.c_void_p),
                    ("kern", C.c_void_p), ("ctx", C.c_void_p)]

    fn()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    cu, graph, n, kind = C.CDLL("libcuda.so.1"), C.c_void_p(g.raw_cuda_graph()), C.c_size_t(0), C.c_int(0)
    assert cu.cuGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, C.byref(n)) == 0
    names = []
    for node in nodes:
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        if kind.value:
            continue
        p, name = Params(), C.c_char_p()
        assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
        if p.func:
            assert cu.cuFuncGetName(C.byref(name), C.c_void_p(p.func)) == 0
        else:
            assert cu.cuKernelGetName(C.byref(name), C.c_void_p(p.kern)) == 0
        names.append(name.value.decode())
    return names


@pytest.mark.parametrize("T,hidden,wide", [(257, 1024, False), (300, 7168, False), (4000, 2048, False), (4000, 4096, False),
                                           (4000, 6144, False), (3999, 6272, False), (4000, 6272, True), (9473, 7168, True)])
def test_columns_of_a_combine_thread(T, hidden, wide):
    """16 columns a thread only where that is the faster form, on both sides of the rule's lines; the last columns of 6272 are a
    quarter of a turn.  Every output kind against the oracle, tokens without a local expert among them."""
    import dataclasses
    from justgoal_b200 import MoELayer
    shape = dataclasses.replace(I.TINY_RENORM, hidden=hidden, num_local_experts=2)
    d = I.make_inputs(shape, T, seed=3)
    layer = MoELayer(shape)
    layer.workspace(T).fill_(0xFF)
    _, out = _forward(shape, d, layer)
    _check_output(shape, d, out)
    dc = util.to_cuda(d)
    idx, w = layer.route(dc["routing_logits"], dc["routing_bias"], dc["routed_scaling_factor"])
    args = (idx, w, dc["hidden_states"], dc["hidden_states_scale"], dc["gemm1_weights"], dc["gemm1_weights_scale"],
            dc["gemm2_weights"], dc["gemm2_weights_scale"], int(d["local_expert_offset"]))
    f32 = layer.forward_routed(*args)
    assert torch.equal(out.view(torch.int16), f32.to(torch.bfloat16).view(torch.int16))
    h16 = layer.forward_routed(*args, out_dtype=torch.float16)
    torch.cuda.synchronize()
    assert layer.status(T) == 0
    assert torch.equal(h16.view(torch.int16), f32.to(torch.float16).view(torch.int16))
    assert bool((out.float() == 0).all(dim=1).any())
    names = [n for n in _kernel_names(lambda: layer.forward(*util.op_args(dc))) if "combine_kernel" in n]
    assert len(names) == 1 and ("combine_kernelILi1ELb%dEE" % wide) in names[0], names


def test_tma_gathered_token_rows_give_the_same_bits():
    """Optional form of GEMM1 for 128-token tiles: the token rows come from hidden_states by four-row TMA gathers
    through the token-of-row table instead of from a gathered copy (no gather launch).  Ragged last tiles, padding
    rows (token -1: the gather reads zeros) and rows of the next expert inside a tile are all in this case."""
    from justgoal_b200 import MoELayer
    shape, T = I.TINY_DS, 600
    d = I.make_inputs(shape, T, seed=91)
    layer = MoELayer(shape)
    assert int(layer.layout(T).token_tile) == 128
    _, out1 = _forward(shape, d, layer)
    out1 = out1.clone()
    n1 = layer.launches_per_forward(T)
    layer.set_tma_gather(True)
    assert layer.launches_per_forward(T) == n1 - 1
    layer.workspace(T).fill_(0xFF)          # stale token ids past the last row must be harmless
    _, out2 = _forward(shape, d, layer)
    assert torch.equal(out1.view(torch.int16), out2.view(torch.int16))
    _check_output(shape, d, out2)


@pytest.mark.parametrize("T", [73, 128, 129])
def test_tma_gathered_token_rows_behind_the_small_front_ends(T):
    """The TMA gather with few tokens (73 is the first count with 128-token tiles here, 128 the last with a one-launch front
    end): GEMM1's producer reads the token-of-row table, so it may not start on the announced routing alone.  Both entry
    points, queued back to back with another call's table still in the workspace, give the bits of the gathered copy."""
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS
    sets = [util.to_cuda(I.make_inputs(shape, T, seed=92 + k)) for k in range(2)]
    layer = MoELayer(shape)
    assert int(layer.layout(T).token_tile) == 128
    wts = ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")
    routed = [layer.route(d["routing_logits"], d["routing_bias"], d["routed_scaling_factor"]) for d in sets]

    def both(k):
        d = sets[k]
        a = layer.forward(*util.op_args(d)).clone()
        b = layer.forward_routed(*routed[k], d["hidden_states"], d["hidden_states_scale"], *[d[n] for n in wts],
                                 int(d["local_expert_offset"]), out_dtype=torch.bfloat16).clone()
        return a, b

    want = [both(k) for k in range(2)]
    layer.set_tma_gather(True)
    layer.workspace(T).fill_(0xFF)
    got = [both(n % 2) for n in range(8)]
    torch.cuda.synchronize()
    assert layer.status(T) == 0
    for n, (a, b) in enumerate(got):
        assert torch.equal(a.view(torch.int16), want[n % 2][0].view(torch.int16)), n
        assert torch.equal(b.view(torch.int16), want[n % 2][1].view(torch.int16)), n


def _kernels_launched(fn):
    """Kernel nodes of the CUDA graph that captures one call of fn."""
    import ctypes as C
    fn()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    cu, graph, n, kind = C.CDLL("libcuda.so.1"), C.c_void_p(g.raw_cuda_graph()), C.c_size_t(0), C.c_int(0)
    assert cu.cuGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, C.byref(n)) == 0
    total = 0
    for node in nodes:
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        total += kind.value == 0                       # CU_GRAPH_NODE_TYPE_KERNEL
    return total


@pytest.mark.parametrize("tma_gather", [False, True])
@pytest.mark.parametrize("T", [40, 128, 129])
def test_launch_counts_are_the_kernels_of_a_captured_call(T, tma_gather):
    """What launches_per_forward, launches_routed and launches_routed_slots state is what a call launches, on both sides of
    the one-launch front ends' limit (40 tokens: narrow tiles; 128 and 129: 128-token tiles, where the TMA gather acts)."""
    from justgoal_b200 import MoELayer
    from justgoal_b200.ep import PeerExchange
    shape = I.TINY_DS
    d = util.to_cuda(I.make_inputs(shape, T, seed=66))
    off = int(d["local_expert_offset"])
    wts = {n: d[n] for n in ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")}
    layer = MoELayer(shape)
    layer.set_tma_gather(tma_gather)
    args = util.op_args(d)
    own = layer.launches_per_forward(T)
    assert own == _kernels_launched(lambda: layer.forward(*args)) == (4 if T <= 128 else 5 if tma_gather else 6)
    if T == 40:
        layer.set_fused_combine(True)
        assert layer.launches_per_forward(T) == _kernels_launched(lambda: layer.forward(*args)) == 3
        layer.set_fused_combine(False)
    idx, w = layer.route(d["routing_logits"], d["routing_bias"], d["routed_scaling_factor"])
    routed = _kernels_launched(lambda: layer.forward_routed(idx, w, d["hidden_states"], d["hidden_states_scale"],
                                                            *wts.values(), off))
    assert layer.launches_routed(T) == routed == (4 if T <= 128 else 5 if tma_gather else 6)
    n = PeerExchange.buffer_bytes(layer, shape, T, 1)
    px = PeerExchange(layer, shape, T, None, None, local_buffers=[torch.zeros(n, dtype=torch.uint8, device="cuda")], rank=0)
    px.wire[:, shape.hidden + 4 * (shape.hidden // 128):].view(torch.int32).fill_(-1)          # empty slots
    slots = _kernels_launched(lambda: px.experts_to_peers(wts, off))
    assert layer.launches_routed_slots(T) == slots == (5 if tma_gather and T > 72 else 6)


def test_workspace_reuse_across_sizes():
    """One layer object, shrinking and growing token counts back to back (workspace buckets, stale
    tables from the larger call must not leak into the smaller one)."""
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS
    layer = MoELayer(shape)
    for T, seed in ((513, 51), (5, 52), (130, 53), (64, 54)):
        d = I.make_inputs(shape, T, seed=seed)
        _, out = _forward(shape, d, layer)
        _check_output(shape, d, out)


def test_ep_combine_kernel_matches_restatement():
    """b200moe_ep_combine: fp32 sum in rank order of the fp16 partial rows a token's ranks sent back."""
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS
    layer = MoELayer(shape)
    T, world, H = 37, 4, shape.hidden
    g = torch.Generator().manual_seed(61)
    has = torch.rand(world, T, generator=g) < 0.6
    has[:, 5] = False                                     # a token nobody computed: zeros
    row_of = torch.full((world, T), -1, dtype=torch.int32)
    row_of[has] = torch.arange(int(has.sum()), dtype=torch.int32)
    back = torch.randn(int(has.sum()), H, generator=g).to(torch.float16)
    got = layer.ep_combine(back.cuda(), row_of.cuda(), T).cpu()
    want = torch.zeros(T, H, dtype=torch.float32)
    for r in range(world):
        sel = row_of[r] >= 0
        want[sel] += back[row_of[r][sel].long()].float()
    assert torch.equal(got.view(torch.int16), want.to(torch.bfloat16).view(torch.int16))
    assert bool((got[5].float() == 0).all())


def test_forward_routed_bf16_and_fp16_are_the_rounded_fp32_result():
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS
    T = 45
    d = util.to_cuda(I.make_inputs(shape, T, seed=62))
    layer = MoELayer(shape)
    idx, w = layer.route(d["routing_logits"], d["routing_bias"], d["routed_scaling_factor"])
    args = (idx, w, d["hidden_states"], d["hidden_states_scale"], d["gemm1_weights"], d["gemm1_weights_scale"],
            d["gemm2_weights"], d["gemm2_weights_scale"], d["local_expert_offset"])
    f32 = layer.forward_routed(*args).clone()
    b16 = layer.forward_routed(*args, out_dtype=torch.bfloat16).clone()
    h16 = layer.forward_routed(*args, out_dtype=torch.float16)
    torch.cuda.synchronize()
    assert torch.equal(b16.view(torch.int16), f32.to(torch.bfloat16).view(torch.int16))
    assert torch.equal(h16.view(torch.int16), f32.to(torch.float16).view(torch.int16))


def test_forward_routed_around_its_front_ends_boundary():
    """Routed calls of 1 to 129 tokens (128 is the last size of the one-launch front end, 32 / 33 its grid sizes), queued
    without a host wait on a poisoned workspace, some ids -1 as on the expert-parallel receive side: each gives the bits of
    the forward that routes itself, apart from the dropped pairs, which the oracle checks."""
    from justgoal_b200 import MoELayer
    shape, sizes = I.TINY_DS, (1, 128, 33, 129, 32, 127)
    d = I.make_inputs(shape, 129, seed=64)
    dc = util.to_cuda(d)
    off = int(d["local_expert_offset"])
    wts = ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")
    layer = MoELayer(shape)
    idx, w = layer.route(dc["routing_logits"], dc["routing_bias"], dc["routed_scaling_factor"])
    drop = idx.clone()
    drop[:, 3] = -1
    for T in sizes:
        layer.workspace(T).fill_(0xFF)
    hs = [(dc["hidden_states"][:T], dc["hidden_states_scale"][:, :T].contiguous()) for T in sizes]
    got = {}
    for k in range(2):
        for T, (x, sc) in zip(sizes, hs):
            for name, ids in (("all", idx), ("drop", drop)):
                out = layer.forward_routed(ids[:T].contiguous(), w[:T].contiguous(), x, sc, *[dc[n] for n in wts], off,
                                           out_dtype=torch.bfloat16).clone()
                if k:
                    assert torch.equal(out.view(torch.int16), got[T, name].view(torch.int16))
                got[T, name] = out
    for T, (x, sc) in zip(sizes, hs):
        assert layer.status(T) == 0
        own = layer.forward(dc["routing_logits"][:T], dc["routing_bias"], x, sc, *[dc[n] for n in wts], off,
                            dc["routed_scaling_factor"])
        assert torch.equal(own.view(torch.int16), got[T, "all"].view(torch.int16))
        want, _, _ = O.run_experts(d["hidden_states"][:T], d["hidden_states_scale"][:, :T].contiguous(), *[d[n] for n in wts],
                                   w[:T].cpu(), drop[:T].cpu().long(), off, shape.num_experts)
        rep = O.compare_output(got[T, "drop"], want.to(torch.bfloat16), util.ATOL, util.RTOL)
        assert rep["finite"] and rep["fail_frac"] == 0.0, (T, rep)


@pytest.mark.parametrize("tile", [0, 16, 128])
@pytest.mark.parametrize("T", [60, 128, 200])
def test_routed_ids_beyond_the_row_capacity_are_refused_whole(T, tile):
    """One local expert and top-8 rows that name it eight times: eight rows a token where the buffers hold one.  The call
    reports error word 5, writes zeros, stores nothing behind the workspace, and the next call on the layer is right.
    (60 and 128 tokens go through the one-launch front end and GEMM1's own tables, 200 through count and permute.)"""
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS.with_local(1)
    d = I.make_inputs(shape, T, seed=65)
    dc = util.to_cuda(d)
    layer = MoELayer(shape)
    layer.set_token_tile(tile)
    bucket = 64 if T <= 64 else 128 if T <= 128 else 256
    used, guard = int(layer.layout(bucket).total_bytes), 1 << 22
    assert 8 * T > int(layer.layout(T).rows_cap)
    ws = torch.full((used + guard,), 0xA5, dtype=torch.uint8, device="cuda")
    layer._ws[bucket] = ws
    idx = torch.zeros(T, shape.top_k, dtype=torch.int32, device="cuda")
    w = torch.rand(T, shape.top_k, generator=torch.Generator().manual_seed(4)).cuda() + 0.1
    wts = [dc[n] for n in ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")]
    for kind in (torch.bfloat16, torch.float32):
        out = torch.full((T, shape.hidden), 7.0, dtype=kind, device="cuda")
        layer.forward_routed(idx, w, dc["hidden_states"], dc["hidden_states_scale"], *wts, 0, output=out)
        torch.cuda.synchronize()
        assert layer.status(T) == 5
        assert bool((out == 0).all()) and bool((ws[used:] == 0xA5).all())
    once = idx.clone()
    once[:, 1:] = shape.num_experts - 1                  # not on this rank
    got = layer.forward_routed(once, w, dc["hidden_states"], dc["hidden_states_scale"], *wts, 0, out_dtype=torch.bfloat16)
    torch.cuda.synchronize()
    assert layer.status(T) == 0
    want, _, _ = O.run_experts(d["hidden_states"], d["hidden_states_scale"], d["gemm1_weights"], d["gemm1_weights_scale"],
                               d["gemm2_weights"], d["gemm2_weights_scale"], w.cpu(), once.cpu().long(), 0, shape.num_experts)
    rep = O.compare_output(got, want.to(torch.bfloat16), util.ATOL, util.RTOL)
    assert rep["finite"] and rep["fail_frac"] == 0.0, rep


def test_ep_pack_unpack_round_trip():
    """b200moe_ep_pack / _unpack: the wire row is [fp8 row | scales | ids | weights] padded to 16 bytes;
    unpacking returns the operator's layouts (scales K-block major) for exactly the packed tokens."""
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS
    T = 50
    d = util.to_cuda(I.make_inputs(shape, T, seed=63))
    layer = MoELayer(shape)
    idx, w = layer.route(d["routing_logits"], d["routing_bias"], d["routed_scaling_factor"])
    send = torch.tensor([3, 3, 49, 0, 17, 20, 21, 48], dtype=torch.int64, device="cuda")
    wire = layer.ep_pack(d["hidden_states"], d["hidden_states_scale"], idx, w, send)
    H, K, KB = shape.hidden, shape.top_k, shape.hidden // 128
    assert wire.shape == (send.numel(), (H + 4 * KB + 8 * K + 15) // 16 * 16) == (send.numel(), layer.ep_row_bytes())
    assert torch.equal(wire[:, :H], d["hidden_states"].view(torch.uint8)[send])
    x, sc, i2, w2 = layer.ep_unpack(wire)
    torch.cuda.synchronize()
    assert torch.equal(x.view(torch.uint8), d["hidden_states"].view(torch.uint8)[send])
    assert torch.equal(sc, d["hidden_states_scale"][:, send])
    assert torch.equal(i2, idx[send]) and torch.equal(w2, w[send])


def test_host_pipeline_returns_every_steps_own_result():
    """HostPipeline overlaps copies and forwards of consecutive steps over two sets of device buffers:
    each step's host output must be that step's own result, bit for bit."""
    from justgoal_b200 import HostPipeline, MoELayer
    shape, T = I.TINY_DS, 40
    layer = MoELayer(shape)
    base = util.to_cuda(I.make_inputs(shape, T, seed=70))
    static = [base[k] for k in ("routing_bias", "gemm1_weights", "gemm1_weights_scale", "gemm2_weights",
                                "gemm2_weights_scale", "local_expert_offset", "routed_scaling_factor")]
    steps = []
    for i in range(5):
        tok = I.make_tokens(shape, T, seed=71 + i, device="cpu")
        steps.append(dict(logits=tok["routing_logits"].pin_memory(), hidden=tok["hidden_states"].pin_memory(),
                          scale=tok["hidden_states_scale"].pin_memory(),
                          out=torch.empty(T, shape.hidden, dtype=torch.bfloat16).pin_memory()))
    pipe = HostPipeline(layer, T, *static)
    for s in steps:
        pipe.step(s["logits"], s["hidden"], s["scale"], s["out"])
    pipe.drain()
    for s in steps:
        want = layer.forward(s["logits"].cuda(), static[0], s["hidden"].cuda(), s["scale"].cuda(), *static[1:])
        torch.cuda.synchronize()
        assert torch.equal(s["out"].view(torch.int16), want.cpu().view(torch.int16))


@pytest.mark.parametrize("tile", [0, 16, 128])
def test_counts_of_the_one_launch_front_ends(tile):
    """The front ends' counts belong to the handle and the last kernel of a forward clears them: own and routed calls on both sides
    of the lines between the grids (8 / 9, 32 / 33 tokens, 128) in turn, queued without a host wait, and the same calls from a
    graph that is replayed, all give the bits of the first pass."""
    from justgoal_b200 import MoELayer
    shape = I.TINY_DS
    d = util.to_cuda(I.make_inputs(shape, 128, seed=67))
    off, f = int(d["local_expert_offset"]), d["routed_scaling_factor"]
    wts = [d[n] for n in ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale")]
    layer = MoELayer(shape)
    layer.set_token_tile(tile)
    idx, w = layer.route(d["routing_logits"], d["routing_bias"], f)
    calls = []
    for T in (8, 128, 9, 1, 33, 32):
        x, sc = d["hidden_states"][:T], d["hidden_states_scale"][:, :T].contiguous()
        layer.workspace(T).fill_(0xFF)
        calls.append(lambda T=T, x=x, sc=sc: layer.forward(d["routing_logits"][:T], d["routing_bias"], x, sc, *wts, off, f))
        calls.append(lambda T=T, x=x, sc=sc: layer.forward_routed(idx[:T], w[:T], x, sc, *wts, off, out_dtype=torch.bfloat16))
    want = [c().clone() for c in calls]
    for own, routed in zip(want[::2], want[1::2]):
        assert torch.equal(own.view(torch.int16), routed.view(torch.int16))
    passes = [[c().clone() for c in calls] for _ in range(3)]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        outs = [c() for c in calls]
    for _ in range(3):
        for o in outs:
            o.fill_(7.0)
        g.replay()
        passes.append([o.clone() for o in outs])
    torch.cuda.synchronize()
    assert [layer.status(T) for T in (1, 8, 9, 32, 33, 128)] == [0] * 6
    for got in passes:
        assert all(torch.equal(a.view(torch.int16), b.view(torch.int16)) for a, b in zip(got, want))
