"""CUDA quantisers vs the oracle: bit-exact bytes and scale bits (through the C ABI)."""
import numpy as np
import pytest
import torch

from oracle import fp8_spec as S

pytestmark = pytest.mark.gpu


def bits(t):
    return t.contiguous().view(torch.uint8 if t.element_size() == 1 else torch.int32).cpu()


@pytest.fixture(scope="module")
def ops(built_library):
    from nano_qwen_b200 import ops
    ops.init()
    return ops


@pytest.mark.parametrize("m,k", [(1, 128), (7, 1024), (16, 4096), (129, 3072), (64, 12288), (300, 256),
                                 (5, 192), (3, 100), (2, 17), (33, 4096 + 64)])
def test_act_quant_bit_exact(ops, m, k):
    g = torch.Generator().manual_seed(m * 1000 + k)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    xq_ref, sx_ref = S.quantize_act_group128(x)
    xq, sx = ops.act_quant(x.cuda())
    torch.cuda.synchronize()
    assert xq.shape == (m, k) and sx.shape == sx_ref.shape
    assert torch.equal(bits(sx), bits(sx_ref))
    assert torch.equal(bits(xq) & 0x7F, bits(xq_ref) & 0x7F)      # sign of an exact zero is not significant
    nz = (bits(xq_ref) & 0x7F) != 0
    assert torch.equal(bits(xq)[nz], bits(xq_ref)[nz])


@pytest.mark.parametrize("m,k,col", [(1, 8, 0), (301, 1096, 0), (3000, 136, 0), (17, 1096, 8), (17, 1096, 4), (9, 1100, 0)])
def test_act_quant_rows_that_end_inside_a_group(ops, m, k, col):
    """Multiples of 8 with 16-byte loads; a start that is not 16-byte aligned and other lengths element by element.
    The bytes between a row's end and the next row are left alone."""
    from nano_qwen_b200 import _cabi
    g = torch.Generator().manual_seed(k + col)
    wide = (torch.randn(m, k + 16, generator=g) * 8.0).to(torch.bfloat16)
    x = wide[:, col:col + k]
    xq_ref, sx_ref = S.quantize_act_group128(x)
    ld = (k + 15) // 16 * 16 + 16
    xq = torch.full((m, ld), 7, dtype=torch.uint8, device="cuda")
    sx = torch.empty(sx_ref.shape[1], m, device="cuda")
    xd = wide.cuda()[:, col:col + k]
    st = _cabi.lib().nq_act_quant_e4m3_g128(xd.data_ptr(), m, k, xd.stride(0), xq.data_ptr(), ld, sx.data_ptr(), m,
                                            torch.cuda.current_stream().cuda_stream)
    assert st == 0
    assert torch.equal(bits(sx.t().contiguous()), bits(sx_ref))
    assert torch.equal(xq[:, :k].cpu() & 0x7F, bits(xq_ref) & 0x7F)
    assert bool((xq[:, k:] == 7).all())


@pytest.mark.parametrize("m,k", [(1, 8), (7, 200), (8, 256)])
def test_quantised_layout_and_leading_dimensions(ops, m, k):
    """Row strides are multiples of 16 bytes, scales are K-group major; a 3-D input gives what its 2-D view gives, on a
    stream of its own too."""
    x = torch.randn(2, m, k, device="cuda").to(torch.bfloat16)
    w = torch.randn(24, k, device="cuda").to(torch.bfloat16)
    xq, sx = ops.act_quant(x[0])
    assert xq.stride() == ((k + 15) // 16 * 16, 1) and sx.stride() == (1, (m + 3) // 4 * 4)
    wq, sw = ops.weight_quant(w)
    flat = ops.fp8_linear(x.view(2 * m, k), wq, sw)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        lead = ops.fp8_linear(x, wq, sw)
        assert ops._stream() == stream.cuda_stream
    stream.synchronize()
    assert lead.shape == (2, m, 24) and torch.equal(lead.view(2 * m, 24), flat)
    assert torch.equal(ops.fp8_gemm(xq, sx, wq, sw), flat[:m])


def test_act_quant_bit_exact_over_many_scales(ops):
    """16 M elements, per-row magnitudes from 2^-60 to 2^60: the reciprocal-based exact division agrees
    with the IEEE divide of the oracle on every byte."""
    g = torch.Generator().manual_seed(2024)
    x = torch.randn(4096, 4096, generator=g)
    x = x * torch.exp2(torch.randint(-60, 61, (4096, 1), generator=g).float()) * (1 + torch.rand(4096, 1, generator=g))
    x = x.to(torch.bfloat16)
    xq_ref, sx_ref = S.quantize_act_group128(x)
    xq, sx = ops.act_quant(x.cuda())
    assert torch.equal(bits(sx), bits(sx_ref))
    assert torch.equal(bits(xq) & 0x7F, bits(xq_ref) & 0x7F)
    nz = (bits(xq_ref) & 0x7F) != 0
    assert torch.equal(bits(xq)[nz], bits(xq_ref)[nz])


def test_act_quant_edge_values(ops):
    x = torch.zeros(6, 256, dtype=torch.bfloat16)
    x[0, :128] = 1.0
    x[0, 128] = 448.0
    x[0, 129] = -3.0
    x[1, 5] = -2.0
    x[3, :] = torch.finfo(torch.bfloat16).max                      # huge values: scale ~7.6e35, q = 448
    x[4, 0], x[4, 1] = 1.0, 2.0 ** -10                             # lands between e4m3 subnormal steps after scaling
    x[5, 0], x[5, 1], x[5, 2] = 1.0, 1.0 / 448 * 2 ** -9 * 1.5, 1e-30    # subnormal midpoint, underflow to zero
    xq_ref, sx_ref = S.quantize_act_group128(x)
    xq, sx = ops.act_quant(x.cuda())
    assert torch.equal(bits(sx), bits(sx_ref))
    assert torch.equal(bits(xq) & 0x7F, bits(xq_ref) & 0x7F)
    assert sx[2, 0].item() == np.float32(1e-10) / np.float32(448)  # all-zero group


def test_act_quant_strided_input_and_large(ops):
    g = torch.Generator().manual_seed(3)
    big = torch.randn(2048, 4096 + 256, generator=g).to(torch.bfloat16)
    view = big[:, 128:128 + 4096]                                  # row stride != K
    xq_ref, sx_ref = S.quantize_act_group128(view)
    xq, sx = ops.act_quant(big.cuda()[:, 128:128 + 4096])
    assert torch.equal(bits(sx), bits(sx_ref))
    assert torch.equal(bits(xq) & 0x7F, bits(xq_ref) & 0x7F)


@pytest.mark.parametrize("n,k", [(128, 128), (1024, 2048), (4096, 1024), (130, 200), (256, 100), (384, 4096 + 64)])
def test_weight_quant_bit_exact(ops, n, k):
    g = torch.Generator().manual_seed(n + k)
    w = (torch.randn(n, k, generator=g) * 0.02).to(torch.bfloat16)
    wq_ref, sw_ref = S.quantize_weight_block128(w)
    wq, sw = ops.weight_quant(w.cuda())
    assert torch.equal(bits(sw), bits(sw_ref))
    assert torch.equal(bits(wq) & 0x7F, bits(wq_ref) & 0x7F)


@pytest.mark.parametrize("n,k,col,ldw,row,ld_wq", [
    (256, 256, 0, 256, 128, 256),        # rows of a merged parameter, 16-byte loads
    (130, 200, 8, 216, 0, 208),          # ragged edges, a column slice of the checkpoint tensor
    (1, 8, 0, 8, 0, 8),                  # the smallest that 16-byte loads take
    (129, 128, 1, 136, 128, 128),        # odd start: element by element
    (200, 131, 0, 131, 0, 144),          # odd row length and stride
    (128, 136, 0, 136, 0, 140),          # rows of the result not 8-byte aligned
])
def test_weight_quant_into_rows_bytes_equal_ieee(ops, n, k, col, ldw, row, ld_wq):
    """Against (w / scale) in IEEE fp32, signs of zeros included, over many binades; nothing outside the rows is written."""
    g = torch.Generator().manual_seed(n + k)
    w = torch.randn(n, k, generator=g) * torch.exp2(torch.randint(-24, 24, (n, 1), generator=g).float())
    w = w.masked_fill(torch.rand(n, k, generator=g) < 0.05, -0.0).to(torch.bfloat16)
    w[:128, :128] = 0.0 if n > 200 else w[:128, :128]                       # an all-zero block
    if n > 128:
        w[128, 0] = float("inf")                                            # scale inf: quotients are zeros and a NaN
    blocks = (-(-n // 128), -(-k // 128))
    wide = torch.zeros(n, ldw, dtype=torch.bfloat16)
    wide[:, col:col + k] = w
    out = torch.full((row + n + 3, ld_wq), 7, dtype=torch.uint8, device="cuda")
    scales = torch.full((row // 128 + blocks[0] + 1, blocks[1]), 7.0, device="cuda")
    dst = out.view(torch.float8_e4m3fn)[row:row + n, :k]
    dst_s = scales[row // 128:row // 128 + blocks[0]]
    assert ops.weight_quant_into(wide.cuda()[:, col:col + k], dst, dst_s)
    padded = torch.zeros(blocks[0] * 128, blocks[1] * 128)
    padded[:n, :k] = w.float()
    amax = padded.view(blocks[0], 128, blocks[1], 128).abs().amax(dim=(1, 3))
    scale = amax.clamp_min(1e-10) / 448.0
    full = scale.repeat_interleave(128, 0).repeat_interleave(128, 1)[:n, :k]
    ref = (w.float() / full)
    want = ref.clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
    got = out.cpu()[row:row + n, :k]
    nan = ref.isnan()
    assert torch.equal(got[~nan], want[~nan]) and bool(((got[nan] & 0x7F) == 0x7F).all())
    assert torch.equal(dst_s.cpu(), scale)
    rest = out.cpu()
    rest[row:row + n, :k] = 7
    assert bool((rest == 7).all()) and bool((scales[row // 128 + blocks[0]:] == 7).all()) and bool((scales[:row // 128] == 7).all())


def test_weight_quant_into_declines_what_it_cannot_write(ops):
    w = torch.randn(128, 256, device="cuda").to(torch.bfloat16)
    q = torch.zeros(128, 256, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    s = torch.zeros(1, 2, device="cuda")
    for wq, sw in ((q[:64], s), (q, s[:, :1]), (q.view(256, 128).t(), s), (q.cpu(), s), (q, s.double())):
        assert not ops.weight_quant_into(w, wq, sw)
    assert not q.view(torch.uint8).any() and not s.any()


def test_quantisers_leave_status_clean(ops):
    from nano_qwen_b200 import _cabi
    torch.cuda.synchronize()
    assert _cabi.device_status()["code"] == 0
