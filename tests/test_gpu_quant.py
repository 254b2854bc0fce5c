"""GPU: the activation quantiser (bf16 -> e4m3 + 1x128 scales, the step before the operator) through the
C ABI, BIT-EXACT against the host statement of the same arithmetic (justgoal_b200.inputs.quantize_rows_1x128:
scale = amax/448 per (token, 128 columns), 1.0 for an all-zero group, round to nearest even)."""
import pytest
import torch

import util
from util import I

pytestmark = pytest.mark.gpu


def _case(T, H, seed, spread=1.0):
    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(T, H, generator=g) * spread).to(torch.bfloat16)
    if T:
        x[0, :128] = 0                      # an all-zero group: scale 1.0, bytes 0
        x[T - 1, H - 128:] *= 1e-3          # a tiny group
        x[T // 2, 5] = 3.0e4                # one large outlier: the rest of its group lands in the subnormals
    return x


@pytest.mark.parametrize("T,H", [(1, 128), (7, 384), (64, 7168), (333, 4096), (4096, 7168)])
def test_quantiser_bit_exact(T, H):
    from justgoal_b200 import quantize_1x128
    x = _case(T, H, seed=T + H)
    q_ref, s_ref = I.quantize_rows_1x128(x)
    q, s = quantize_1x128(x.cuda())
    torch.cuda.synchronize()
    assert s.shape == (H // 128, T) and q.shape == (T, H)
    assert torch.equal(s.cpu().view(torch.int32), s_ref.view(torch.int32))
    assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))


@pytest.mark.parametrize("spread", [1.0, 2.0 ** -88, 2.0 ** -120, 2.0 ** 119])
def test_quantiser_every_pair_of_mantissas(spread):
    """The kernel's quotients are corrected products, not divisions: every pair of bf16 mantissas (group maximum, element)
    at every exponent gap that still reaches the e4m3 grid gives the byte of the IEEE division; tiny and huge scales too."""
    from justgoal_b200 import quantize_1x128
    m = 1.0 + torch.arange(128, dtype=torch.float64) / 128
    gaps = 2.0 ** -torch.arange(0, 20, dtype=torch.float64)
    x = (m[None, None, :] * gaps[None, :, None] * 0.5).repeat(128, 1, 1)         # [maximum, gap, element], elements below the maximum
    x = (x * spread).to(torch.bfloat16).clone()
    x[:, :, ::3] *= -1
    tail = x[:, :, 127].clone()
    x[:, :, 127] = (m * spread).to(torch.bfloat16)[:, None]             # the group's maximum
    x[:, :, 64] = tail                                                  # (element 64 gives way to the one the maximum displaced)
    x = x.reshape(128 * 20, 128)
    x = torch.cat([x, x.flip(0)], dim=1).contiguous()
    q_ref, s_ref = I.quantize_rows_1x128(x)
    q, s = quantize_1x128(x.cuda())
    assert torch.equal(s.cpu().view(torch.int32), s_ref.view(torch.int32))
    assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -88, 2.0 ** -120, 2.0 ** 119])
def test_quantiser_keeps_the_sign_of_zeros_and_of_underflow(scale):
    """-0 becomes the byte 0x80 and +0 the byte 0x00, in a group of zeros, in an ordinary group and where the division is
    taken instead of the product; elements far below the e4m3 grid round to the zero of their own sign."""
    from justgoal_b200 import quantize_1x128
    x = torch.zeros(9, 384)
    x[:, 0:128:2] = -0.0                                            # zeros of both signs alone: scale 1
    x[:, 128:256] = torch.randn(9, 128, generator=torch.Generator().manual_seed(6)) * scale
    x[:, 130:250:7], x[:, 131:250:7] = -0.0, 0.0
    x[:, 256:384] = torch.tensor([1.0, -1.0]).repeat(64) * scale * 2.0 ** -torch.arange(14, 23).float()[:, None]
    x[:, 256] = scale                                               # the group's maximum; the others reach the grid's end
    x = x.to(torch.bfloat16)
    q_ref, s_ref = I.quantize_rows_1x128(x)
    want = q_ref.view(torch.uint8)
    zeros = x.float() == 0
    negative = torch.signbit(x.float())
    assert bool((want[zeros & negative] == 0x80).all()) and bool((want[zeros & ~negative] == 0).all())
    q, s = quantize_1x128(x.cuda())
    assert torch.equal(s.cpu().view(torch.int32), s_ref.view(torch.int32))
    assert torch.equal(q.cpu().view(torch.uint8), want)


@pytest.mark.parametrize("T,H,off", [(1, 128, 0), (9, 256, 8), (31, 4352, 8), (600, 8320, 0), (4739, 128, 16), (40003, 128, 0),
                                     (19001, 384, 8), (9999, 512, 16)])
def test_quantiser_blocks_and_alignment(T, H, off):
    """Ragged token blocks, rows cut over several CTAs, rows of few groups (up to 64 tokens in a CTA), and activations that are
    only 16-byte aligned."""
    from justgoal_b200 import _lib, quantize_1x128
    import ctypes as C
    x = _case(T, H, seed=T)
    buf = torch.zeros(T * H + 16, dtype=torch.bfloat16, device="cuda")
    view = buf[off:off + T * H].view(T, H)
    view.copy_(x)
    q_ref, s_ref = I.quantize_rows_1x128(x)
    q, s = quantize_1x128(view)
    assert torch.equal(s.cpu().view(torch.int32), s_ref.view(torch.int32))
    assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))
    qb = torch.zeros(T * H + 8, dtype=torch.uint8, device="cuda")       # output that is only 8-byte aligned
    rc = _lib.lib.b200moe_quantize_1x128(C.c_void_p(view.data_ptr()), T, H, C.c_void_p(qb.data_ptr() + 8), C.c_void_p(s.data_ptr()), None)
    torch.cuda.synchronize()
    assert rc == 0 and torch.equal(qb[8:].cpu().view(T, H), q_ref.view(torch.uint8))


@pytest.mark.parametrize("T,H", [(9471, 2048), (9473, 2048), (2369, 2048), (9472, 1024), (1187, 7168)])
def test_quantiser_tokens_of_a_cta(T, H):
    """Both sides of the lines between two, four and eight tokens per CTA (eight CTAs per SM of eight tokens, two of four), and rows of
    few groups, whose CTAs keep eight."""
    from justgoal_b200 import quantize_1x128
    x = _case(T, H, seed=T)
    q_ref, s_ref = I.quantize_rows_1x128(x)
    q, s = quantize_1x128(x.cuda())
    torch.cuda.synchronize()
    assert torch.equal(s.cpu().view(torch.int32), s_ref.view(torch.int32))
    assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))


def test_quantiser_between_its_neighbours():
    """The quantiser may start under the kernel that writes its input and lets the layer start under itself: a chain of copy,
    quantiser, quantiser into the same input's other half and forward, queued without a host wait, gives the bytes of each call made
    alone."""
    from justgoal_b200 import MoELayer, quantize_1x128
    shape, T = I.TINY_DS, 128
    d = util.to_cuda(I.make_inputs(shape, T, seed=12))
    layer = MoELayer(shape)
    rest = [d[n] for n in ("gemm1_weights", "gemm1_weights_scale", "gemm2_weights", "gemm2_weights_scale", "local_expert_offset",
                           "routed_scaling_factor")]
    src = [_case(T, shape.hidden, seed=k).cuda() for k in range(3)]
    want = []
    for x in src:
        q, s = quantize_1x128(x)
        torch.cuda.synchronize()
        out = layer.forward(d["routing_logits"], d["routing_bias"], q, s, *rest).clone()
        torch.cuda.synchronize()
        want.append((q.view(torch.uint8).clone(), s.clone(), out))
    x, got = torch.empty_like(src[0]), []
    for k in range(12):
        x.copy_(src[k % 3])
        q, s = quantize_1x128(x)
        x.fill_(100.0)
        quantize_1x128(x)
        got.append((q.view(torch.uint8), s, layer.forward(d["routing_logits"], d["routing_bias"], q, s, *rest)))
    torch.cuda.synchronize()
    for k, (q, s, out) in enumerate(got):
        assert torch.equal(q, want[k % 3][0]) and torch.equal(s, want[k % 3][1])
        assert torch.equal(out.view(torch.int16), want[k % 3][2].view(torch.int16))


def test_quantiser_feeds_the_operator():
    """bf16 activations -> quantiser kernel -> layer: same output as with host-quantised inputs."""
    from justgoal_b200 import MoELayer, quantize_1x128
    shape = I.TINY_DS
    d = I.make_inputs(shape, 50, seed=77)
    x = torch.randn(50, shape.hidden, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16)
    d["hidden_states"], d["hidden_states_scale"] = I.quantize_rows_1x128(x)
    dc = util.to_cuda(d)
    layer = MoELayer(shape)
    want = layer.forward(*util.op_args(dc)).clone()
    dc["hidden_states"], dc["hidden_states_scale"] = quantize_1x128(x.cuda())
    got = layer.forward(*util.op_args(dc))
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    rep = util.O.compare_output(got, util.run_oracle(shape, d).output, util.ATOL, util.RTOL)
    assert rep["fail_frac"] == 0.0, rep


def test_quantiser_rejects_bad_shapes():
    from justgoal_b200 import _lib
    assert _lib.lib.b200moe_quantize_1x128(None, 4, 100, None, None, None) == -1      # H not a multiple of 128
    assert _lib.lib.b200moe_quantize_1x128(None, 4, 128, None, None, None) == -1      # null pointers
    assert _lib.lib.b200moe_quantize_1x128(None, 0, 128, None, None, None) == 0       # nothing to do
