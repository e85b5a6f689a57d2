"""The native quantizer (pe_quantize) against the CPU oracle of the reference's quantize_tensor
(quantizer.py:178-257): norms equal to within one fp16 step, codes equal except where a rotated value sits on a
cell boundary to within fp32 rounding (bounded flip rate, every flip to a neighbouring level), and the
dequantised weights equally close to the original."""
import pytest
import torch

import polar_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [2, 3, 4, 5, 6, 8])
def test_gpu_quantizer_matches_the_cpu_order(bits):
    from polarengine_vllm_b200.quantizer import PolarQuantizer
    g = torch.Generator().manual_seed(bits)
    w = torch.randn(512, 1000, generator=g) * 0.02     # ragged K: pads to 1024
    w[7] = 0                                            # an all-zero row: norm clamps at 1e-10
    ref = oracle.quantize_tensor(w, bits)
    q = PolarQuantizer().quantize_tensor_gpu(w.cuda(), bits)
    codes, norms = q["codes"].cpu(), q["norms"].cpu()
    assert codes.shape == ref["codes"].shape and codes.dtype == torch.int8 and norms.dtype == torch.float16
    assert torch.equal(q["ct_scaled"].cpu(), ref["ct_scaled"])
    # norms: the sum of squares is taken in another order
    assert ((norms.float() - ref["norms"].float()).abs() <= ref["norms"].float().abs() * 2 ** -10 + 1e-12).all()
    live = torch.ones(512, dtype=torch.bool); live[7] = False   # codes of a zero block are noise around 0 either way
    diff = (codes[live].view(torch.uint8).int() - ref["codes"][live].view(torch.uint8).int()).abs()
    flips = int((diff != 0).sum())
    assert flips <= max(8, int(2e-5 * diff.numel())), f"{flips} of {diff.numel()} codes differ"
    assert int(diff.max()) <= 1                                  # and only to the neighbouring level
    a = oracle.dequant_fp32(codes, norms, q["ct_scaled"].cpu())[:, :1000]
    b = oracle.dequant_fp32(ref["codes"], ref["norms"], ref["ct_scaled"])[:, :1000]
    ea, eb = float((a - w).norm() / w.norm()), float((b - w).norm() / w.norm())
    assert abs(ea - eb) <= 1e-4 * max(eb, 1e-6) + 1e-6


def test_gpu_quantizer_half_and_bf16_inputs():
    from polarengine_vllm_b200.quantizer import PolarQuantizer
    g = torch.Generator().manual_seed(1)
    w = (torch.randn(64, 384, generator=g) * 0.02)
    for dt in (torch.float16, torch.bfloat16):
        wd = w.to(dt)
        ref = oracle.quantize_tensor(wd.float(), 4)
        q = PolarQuantizer().quantize_tensor_gpu(wd.cuda(), 4)
        assert (q["codes"].cpu() != ref["codes"]).float().mean() < 1e-3


@pytest.mark.parametrize("levels", ["two", "odd", "crowded", "unsorted"])
def test_gpu_quantizer_levels_of_any_kind(levels):
    """Few levels, several edges in one cell of the lookup grid, levels too close together or out of order (scanned)."""
    from polarengine_vllm_b200 import _native as nv
    g = torch.Generator().manual_seed(5)
    lv = {"two": torch.tensor([-0.8, 0.8]), "odd": torch.tensor([-2.0, -0.5, 0.1, 0.4, 3.0]),
          "crowded": torch.cat([torch.linspace(-0.02, 0.02, 40), torch.tensor([5.0, 9.0])]),
          "unsorted": torch.tensor([1.5, -1.5, 0.4, -0.4])}[levels]
    w = torch.randn(33, 200, generator=g) * 0.02
    nv.ensure_init(torch.device("cuda", 0))
    wd, ld = w.cuda(), lv.cuda()
    codes = torch.empty(33, 256, dtype=torch.int8, device="cuda")
    norms = torch.empty(33, 2, dtype=torch.float16, device="cuda")
    nv.check(nv.lib().pe_quantize(wd.data_ptr(), nv.PE_F32, 200, 33, 200, 256, ld.data_ptr(), ld.numel(), codes.data_ptr(), 256,
                                  norms.data_ptr(), 2, nv.stream_ptr(wd.device)), "pe_quantize")
    blocks = torch.nn.functional.pad(w, (0, 56)).view(33, 2, 128)
    rot = blocks / blocks.norm(dim=2, keepdim=True) @ oracle.hadamard(128) * 128 ** 0.5
    ref = (rot.unsqueeze(-1) - lv).abs().argmin(-1).view(33, 256)
    assert int((codes.cpu().view(torch.uint8).int() != ref).sum()) <= 8


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,cols,bits", [(1, 8, 3), (3, 129, 4), (65, 1000, 5), (33, 1152, 6), (130, 4100, 8)])
def test_gpu_quantizer_16_bit_weights(dtype, rows, cols, bits):
    """16-bit weights of any width, row stride and address, an all-zero block among them: the codes that 64-bit arithmetic gives
    except next to a cell edge (a value within 2e-6 of it: fp32 sums of 128 values of order one), the norms to one fp16 step."""
    from polarengine_vllm_b200 import _native as nv
    from polarengine_vllm_b200.utils import get_centroids
    g = torch.Generator().manual_seed(rows + bits)
    wide = (0.02 * torch.randn(rows, cols + 5, generator=g)).to(dtype).cuda()
    wide[0, :128] = 0
    lv, padded = get_centroids(bits).cuda(), -(-cols // 128) * 128
    nv.ensure_init(wide.device)
    out = []
    for w, ld in ((wide[:, :cols].contiguous(), cols), (wide[:, 3:3 + cols], cols + 5)):
        codes = torch.full((rows, padded), 0x55, dtype=torch.int8, device="cuda")
        norms = torch.empty(rows, padded // 128, dtype=torch.float16, device="cuda")
        nv.check(nv.lib().pe_quantize(w.data_ptr(), nv.dtype_code(w), ld, rows, cols, padded, lv.data_ptr(), lv.numel(), codes.data_ptr(), padded,
                                      norms.data_ptr(), padded // 128, nv.stream_ptr(w.device)), "pe_quantize")
        x = torch.nn.functional.pad(w.double(), (0, padded - cols)).view(-1, 128)
        n = x.norm(dim=1).clamp_min(1e-10)
        rot = (x / n[:, None]) @ oracle.hadamard(128).double().cuda() * 128 ** 0.5
        c = codes.view(torch.uint8).long().view(-1, 128)
        excess = (rot - lv.double()[c]).abs() - (rot.unsqueeze(-1) - lv.double()).abs().amin(-1)
        assert float(excess.max()) <= 2e-6
        assert ((norms.double().view(-1) - n).abs() <= n * 2 ** -10 + 1e-7).all()


def test_gpu_quantizer_extreme_values():
    """bf16 values whose squares overflow fp32, infinities and NaN: code 0 where a block has no finite unit vector, its neighbours
    as without it."""
    from polarengine_vllm_b200.quantizer import PolarQuantizer
    g = torch.Generator().manual_seed(3)
    w = (0.02 * torch.randn(4, 1024, generator=g)).to(torch.bfloat16).cuda()
    ref = PolarQuantizer().quantize_tensor_gpu(w, 4)["codes"].view(4, 8, 128)
    x = w.clone()
    x[0, 128:256] *= 2.0 ** 66     # norm about 1.7e19: its square overflows on the way, the norm does not
    x[1, 300], x[2, 5], x[3, 1000] = float("inf"), float("nan"), float("-inf")
    q = PolarQuantizer().quantize_tensor_gpu(x, 4)
    codes, norms = q["codes"].view(4, 8, 128), q["norms"]
    assert torch.equal(codes[0], ref[0]) and bool(torch.isinf(norms[0, 1]))
    for r, b in ((1, 2), (2, 0), (3, 7)):
        assert not codes[r, b].any()
        codes[r, b] = ref[r, b]
    assert torch.equal(codes, ref)


@pytest.mark.parametrize("bits", [3, 4, 6, 8])
def test_gpu_quantizer_sums_beyond_fp32(bits):
    """Finite bf16 blocks whose rotated values are past the largest fp32 number: an infinite norm and the codes of zero, as 32-bit
    weights of the same values give them; the blocks beside them and those just below the line as ever."""
    from polarengine_vllm_b200.quantizer import PolarQuantizer
    g = torch.Generator().manual_seed(bits)
    w = (0.02 * torch.randn(6, 640, generator=g)).to(torch.bfloat16).cuda()
    top = torch.finfo(torch.bfloat16).max
    x = w.clone()
    x[0, :128] = top                                   # one rotated value of 128 times the largest, the others cancel
    x[1, 128:256] = top * torch.sign(w[1, 128:256])    # sums of both signs
    x[2, 256:272] = -top                               # sixteen neighbours
    x[3, 384:512:8] = top                              # sixteen values that are added first
    x[4, 512:640] = 2.0 ** 125 * torch.sign(w[4, 512:640])
    x[5, 5] = top                                      # a single one: no sum is too large, its square is
    q, ref = (PolarQuantizer().quantize_tensor_gpu(t, bits) for t in (x, x.float()))
    assert torch.isinf(q["norms"]).sum() == 6
    assert torch.equal(q["norms"].isinf(), ref["norms"].isinf())
    zero = PolarQuantizer().quantize_tensor_gpu(torch.zeros_like(x[:1]), bits)["codes"][0, 0]
    assert bool((q["codes"].view(6, 5, 128)[q["norms"].isinf()] == zero).all())
    plain = PolarQuantizer().quantize_tensor_gpu(w, bits)
    same = ~q["norms"].isinf()
    assert torch.equal(q["codes"].view(6, 5, 128)[same], plain["codes"].view(6, 5, 128)[same]) and torch.equal(q["norms"][same], plain["norms"][same])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gpu_quantizer_several_infinities_in_a_block(dtype):
    """Infinities that meet in one sum of the rotation, of one sign or both, beside a NaN: code 0 for the block and the norm that
    32-bit weights of the same values get."""
    from polarengine_vllm_b200.quantizer import PolarQuantizer
    inf, nan = float("inf"), float("nan")
    g = torch.Generator().manual_seed(2)
    w = (0.02 * torch.randn(5, 200, generator=g)).to(dtype).cuda()
    x = w.clone()
    for row, at in enumerate([{5: inf, 13: inf}, {5: inf, 21: -inf}, {0: inf, 1: inf, 2: inf, 3: inf}, {7: nan, 71: inf}, {130: -inf, 199: -inf}]):
        for i, v in at.items():
            x[row, i] = v
    q, ref, plain = (PolarQuantizer().quantize_tensor_gpu(t, 4) for t in (x, x.float(), w))
    hit = torch.zeros(5, 2, dtype=torch.bool, device="cuda")
    hit[:4, 0], hit[4, 1] = True, True
    codes = q["codes"].view(5, 2, 128)
    assert not codes[hit].any() and torch.equal(codes[~hit], plain["codes"].view(5, 2, 128)[~hit])
    assert torch.equal(q["norms"], torch.where(hit, ref["norms"], plain["norms"]))
