"""Parity of the tcgen05 prefill kernel (pe_gemm, through the C ABI) with the CPU oracle.
bf16 operands, fp32 accumulation: max |y - ref| / max |ref| <= 1e-2 against the fp32
dequant reference, cosine > 0.9999."""
import pytest
import torch

import polar_oracle as oracle
from helpers import max_rel, rand_layer, rand_x, ref_metrics

pytestmark = pytest.mark.gpu
TOL = 1e-2


def run_gemm(codes, norms, cts, x, bits, rotated=False, out_dtype=torch.float16, bias=None, in_f=None):
    from polarengine_vllm_b200 import _native as nv, gemm, packing
    dev = torch.device("cuda")
    nv.ensure_init(dev)
    n, kp = codes.shape
    packed = bits <= 4
    cd = codes.to(dev)
    w = packing.pack_codes_half_block(cd) if packed else cd
    xd = x.to(dev).contiguous()
    y = torch.full((x.shape[0], n), float("nan"), dtype=out_dtype, device=dev)
    gemm.quant_gemm(w, packed, norms.to(dev), cts.to(dev), xd, rotated, n, in_f if in_f is not None else kp, kp, y,
                    bias.to(dev).half() if bias is not None else None, check_status=True)
    return y


@pytest.mark.parametrize("bits", [3, 4, 5, 6])
@pytest.mark.parametrize("m,n,k", [(64, 256, 256), (256, 512, 1024), (128, 256, 128), (300, 1856, 2688),
                                   (100, 2688, 1920), (17, 130, 384), (1024, 4096, 4096),
                                   (64, 40000, 256)])  # the last: more 256-row tiles than SMs, several tiles per CTA
def test_gemm_matches_oracle(m, n, k, bits):
    codes, norms, cts = rand_layer(n, k, bits, seed=m + n + bits)
    x = rand_x(m, k, seed=3, dtype=torch.bfloat16)
    ref = oracle.linear_dequant(x, codes, norms, cts)
    y = run_gemm(codes, norms, cts, x, bits)
    assert y.shape == (m, n) and torch.isfinite(y.float()).all()
    assert max_rel(y, ref) <= TOL
    cos, _ = ref_metrics(y, ref)
    assert cos > 0.9999


@pytest.mark.parametrize("bits,n,k", [(4, 4096, 4096), (4, 12288, 4096), (4, 4096, 12288), (5, 4096, 4096), (6, 4096, 4096),
                                      (3, 12288, 4096)])
def test_gemm_prefill_sweep_shapes_m4096(bits, n, k):
    """The prefill sweep's largest case: 4096 bf16 tokens into the decoder-layer shapes (the reference's own
    self-test list is polar_gemm.py:541-615).  The kernel runs all 4096 tokens; the CPU oracle is evaluated
    on every 16th token (all output columns), which covers every token tile and every weight tile."""
    m = 4096
    codes, norms, cts = rand_layer(n, k, bits, seed=n + k + bits)
    x = rand_x(m, k, seed=12, dtype=torch.bfloat16)
    y = run_gemm(codes, norms, cts, x, bits)
    assert y.shape == (m, n) and torch.isfinite(y.float()).all()
    rows = torch.arange(5, m, 16)
    ref = oracle.linear_dequant(x[rows], codes, norms, cts)
    assert max_rel(y[rows.cuda()], ref) <= TOL
    cos, _ = ref_metrics(y[rows.cuda()], ref)
    assert cos > 0.9999
    # the first and the last token tile in full
    edge = torch.cat([torch.arange(0, 64), torch.arange(m - 64, m)])
    assert max_rel(y[edge.cuda()], oracle.linear_dequant(x[edge], codes, norms, cts)) <= TOL


def test_gemm_ragged_in_features_bias_and_dtypes():
    n, k, in_f, bits, m = 512, 1920, 1856, 4, 200
    codes, norms, cts = rand_layer(n, k, bits, seed=9)
    bias = rand_x(1, n, seed=4).reshape(n)
    for xdt in (torch.float16, torch.bfloat16, torch.float32):
        x = rand_x(m, in_f, seed=5, dtype=xdt)
        ref = oracle.linear_dequant(x, codes, norms, cts, in_f=in_f) + bias.float()
        for ydt in (torch.float16, torch.bfloat16, torch.float32):
            y = run_gemm(codes, norms, cts, x, bits, out_dtype=ydt, bias=bias, in_f=in_f)
            assert y.dtype == ydt and max_rel(y, ref) <= TOL


@pytest.mark.parametrize("m,n", [(257, 256), (700, 1000), (513, 2688), (1100, 130)])
def test_gemm_some_hundred_rows_ragged_edges_bias_and_dtypes(m, n):
    """A few tiles of tokens on the tensor-memory kernel: token and weight-row counts off every tile and
    vector boundary, padded K, bias, all output types."""
    k, in_f, bits = 1920, 1856, 4
    codes, norms, cts = rand_layer(n, k, bits, seed=m + n)
    bias = rand_x(1, n, seed=4).reshape(n)
    x = rand_x(m, in_f, seed=5, dtype=torch.bfloat16)
    ref = oracle.linear_dequant(x, codes, norms, cts, in_f=in_f) + bias.float()
    for ydt in (torch.float16, torch.bfloat16, torch.float32):
        y = run_gemm(codes, norms, cts, x, bits, out_dtype=ydt, bias=bias, in_f=in_f)
        assert y.dtype == ydt and y.shape == (m, n) and max_rel(y, ref) <= TOL
    y5 = run_gemm(*rand_layer(n, k, 5, seed=n)[:3], x, 5, in_f=in_f)
    c5, n5, t5 = rand_layer(n, k, 5, seed=n)
    assert max_rel(y5, oracle.linear_dequant(x, c5, n5, t5, in_f=in_f)) <= TOL


@pytest.mark.parametrize("m,n", [(4097, 130), (4200, 1000), (4353, 2689), (4097, 37 * 256 + 101)])
def test_gemm_paired_ctas_ragged_edges_bias_and_dtypes(m, n):
    """More than 4096 tokens always run on pairs of CTAs (512-token tiles, each CTA decoding half of the weight tile)
    with the output leaving through clipped TMA stores where its rows are whole 16 bytes: token and weight-row counts off every tile, box and
    vector boundary, padded K, bias, all output types; tiles whole, all of them in K ranges (130 rows) or those of a last wave (2689)."""
    k, in_f = 1920, 1856
    bias = rand_x(1, n, seed=4).reshape(n)
    x = rand_x(m, in_f, seed=5, dtype=torch.bfloat16)
    rows = torch.cat([torch.arange(0, m, 61), torch.arange(m - 20, m)])
    for bits in (4, 5):
        codes, norms, cts = rand_layer(n, k, bits, seed=m + n)
        ref = oracle.linear_dequant(x[rows], codes, norms, cts, in_f=in_f) + bias.float()
        for ydt in (torch.float16, torch.bfloat16, torch.float32):
            y = run_gemm(codes, norms, cts, x, bits, out_dtype=ydt, bias=bias, in_f=in_f)
            assert y.dtype == ydt and y.shape == (m, n) and torch.isfinite(y.float()).all() and max_rel(y[rows.cuda()], ref) <= TOL


def test_gemm_few_tiles_with_and_without_room_for_the_k_split():
    """A launch of up to 256 rows on few 256-row tiles splits K over the SMs when the workspace holds the fp32
    partials (pe_gemm_workspace_bytes_splitk) and runs unsplit in a workspace of pe_gemm_workspace_bytes: same
    values either way (only the order of the fp32 sums differs), bias and output type included."""
    from polarengine_vllm_b200 import _native as nv, packing
    dev = torch.device("cuda")
    nv.ensure_init(dev)
    m, n, k, bits = 96, 1024, 4096, 4
    codes, norms, cts = rand_layer(n, k, bits, seed=31)
    bias = rand_x(1, n, seed=2).reshape(n)
    x = rand_x(m, k, seed=8, dtype=torch.bfloat16)
    ref = oracle.linear_dequant(x, codes, norms, cts) + bias.float()
    w = packing.pack_codes_half_block(codes.to(dev))
    nd, ctd, xd, bd = norms.to(dev), cts.to(dev), x.to(dev), bias.to(dev).half()
    l = nv.lib()
    small, large = l.pe_gemm_workspace_bytes(m, k), l.pe_gemm_workspace_bytes_splitk(m, n, k)
    assert large > small
    out = []
    for size in (small, large):
        ws = torch.zeros(size, dtype=torch.uint8, device=dev)
        y = torch.full((m, n), float("nan"), dtype=torch.float16, device=dev)
        nv.check(l.pe_gemm(w.data_ptr(), 1, w.stride(0), nd.data_ptr(), nd.stride(0), ctd.data_ptr(), ctd.numel(), xd.data_ptr(),
                           nv.PE_X_RAW, nv.dtype_code(xd), xd.stride(0), k, y.data_ptr(), nv.dtype_code(y), y.stride(0),
                           bd.data_ptr(), m, n, k, ws.data_ptr(), ws.numel(), nv.stream_ptr(dev)), "pe_gemm")
        torch.cuda.synchronize()
        assert int(ws[:4].view(torch.int32).item()) == 0
        assert max_rel(y, ref) <= TOL
        out.append(y.float())
    assert max_rel(out[0], out[1]) <= 2e-3


def test_gemm_rotated_input_and_reference_signature():
    """polar_gemm / polar_gemm_packed of the reference take fp32 x_transformed
    (polar_gemm.py:312-418) and agree with the decode kernel (reference self-test
    polar_gemm.py:680-718 bounds the GEMM-vs-GEMV difference)."""
    from polarengine_vllm_b200 import kernels
    n, k, bits, m = 1024, 4096, 4, 64
    codes, norms, cts = rand_layer(n, k, bits, seed=21)
    xt = oracle.fwht(rand_x(m, k, seed=6, dtype=torch.float32))
    cd, nd, ctd, xd = codes.cuda(), norms.cuda(), cts.cuda(), xt.cuda()
    pk = kernels.pack_codes_int4(cd)
    y = kernels.polar_gemm_packed(pk, xd, nd, ctd, n, k // 2, k // 128)
    y_unpacked = kernels.polar_gemm(cd, xd, nd, ctd, n, k, k // 128)
    ref = torch.einsum("rnk,mnk->mr", cts[codes.long()].view(n, -1, 128) * norms.float().view(n, -1, 1), xt.view(m, -1, 128))
    assert y.dtype == torch.float32 and y.shape == (m, n)
    assert max_rel(y, ref) <= TOL and max_rel(y_unpacked, ref) <= TOL
    y_gemv = torch.cat([kernels.polar_matmul(None, xd[i], nd, ctd, n, k, k // 128, 128, True, pk, k // 2).reshape(1, n)
                        for i in range(4)])
    assert max_rel(y[:4], y_gemv) <= TOL


def test_apply_prefill_matches_oracle():
    from polarengine_vllm_b200.linear_method import PolarQuantLinearMethod
    bits, n, in_f = 4, 1024, 1856
    g = torch.Generator().manual_seed(2)
    w = torch.randn(n, in_f, generator=g) * 0.02
    q = oracle.quantize_tensor(w, bits)
    m = PolarQuantLinearMethod(128, bits)
    layer = torch.nn.Module()
    m.create_weights(layer, in_f, [n], in_f, n, torch.float16)
    layer.codes.data.copy_(q["codes"]); layer.norms.data.copy_(q["norms"])
    layer = layer.cuda()
    m.process_weights_after_loading(layer)
    x = rand_x(96, in_f, seed=1).reshape(2, 48, in_f)
    y = m.apply(layer, x.cuda())
    ref = oracle.apply_forward(x, q["codes"], q["norms"], q["ct_scaled"], in_f)
    assert y.shape == (2, 48, n) and y.dtype == torch.float16 and max_rel(y, ref) <= TOL


@pytest.mark.parametrize("m", [17, 32, 129, 191, 192, 193, 256])
@pytest.mark.parametrize("bits,n,k", [(3, 127, 128), (4, 129, 384), (6, 300, 640), (4, 19000, 256), (3, 5000, 1920)])
def test_gemm_up_to_256_rows_edges(m, bits, n, k):
    """Edges of the tensor-memory kernel: token counts around 16, 128 and 192 (two halves), weight rows around 128 and more
    tiles than SMs, an odd number of K blocks, one block (no split), rows at odd addresses, every output type."""
    codes, norms, cts = rand_layer(n, k, bits, seed=m + n)
    in_f = k - 5
    x = rand_x(m, in_f, seed=m)
    ref = oracle.linear_dequant(x, codes, norms, cts, in_f=in_f)
    bias = rand_x(1, n, seed=4).reshape(n)
    for dt in (torch.float16, torch.float32, torch.bfloat16):
        y = run_gemm(codes, norms, cts, x, bits, out_dtype=dt, bias=bias, in_f=in_f)
        assert max_rel(y, ref + bias.float()) <= TOL
    xt = oracle.fwht(torch.nn.functional.pad(x.float(), (0, k - in_f)))
    assert max_rel(run_gemm(codes, norms, cts, xt, bits, rotated=True, in_f=in_f), ref) <= TOL


@pytest.mark.parametrize("m,in_f", [(17, 300), (200, 304), (513, 384)])
def test_gemm_of_gate_up_equals_activation_then_gemm(m, in_f):
    """PE_X_SILU_MUL input: the bits of pe_silu_mul's rounding followed by the same launch, ragged and unaligned widths."""
    from polarengine_vllm_b200 import _native as nv, packing
    n, k = 260, 384
    codes, norms, cts = rand_layer(n, k, 4, seed=m)
    w, nd, ctd = packing.pack_codes_half_block(codes.cuda()), norms.cuda(), cts.cuda()
    gu = rand_x(m, 2 * in_f, seed=in_f).cuda()
    act = torch.nn.functional.silu(gu[:, :in_f]) * gu[:, in_f:]
    y, ref = ((nv._host or nv.host()).matmul(w, True, nd, ctd, x, kind, n, in_f, k, torch.float32, None, None)
              for x, kind in ((gu, nv.PE_X_SILU_MUL), (act, False)))
    assert y is not None and max_rel(y, ref) <= 2e-3
    assert max_rel(y, oracle.linear_dequant(act.cpu(), codes, norms, cts, in_f=in_f)) <= TOL


def with_and_without_room(m, n, k, bits, dtype):
    """The launch with the workspace it would like and with the smallest one, a bias in both; some rows of it from the oracle."""
    from polarengine_vllm_b200 import _native as nv, packing
    codes, norms, cts = rand_layer(n, k, bits, seed=m)
    x, bias = rand_x(m, k, seed=m + 1), rand_x(1, n, seed=2).reshape(n)
    w, packed = (packing.pack_codes_half_block(codes.cuda()), True) if bits <= 4 else (codes.cuda(), False)
    nd, ctd, xd, bd = norms.cuda(), cts.cuda(), x.cuda(), bias.cuda()
    lib, out = nv.lib(), []
    for room in (lib.pe_gemm_workspace_bytes_splitk(m, n, k), lib.pe_gemm_workspace_bytes(m, k)):
        y = torch.full((m, n), float("nan"), dtype=dtype, device="cuda")
        ws = torch.empty(room, dtype=torch.uint8, device="cuda")
        nv.check(lib.pe_gemm(w.data_ptr(), int(packed), w.stride(0), nd.data_ptr(), nd.stride(0), ctd.data_ptr(), ctd.numel(), xd.data_ptr(),
                             nv.PE_X_RAW, nv.dtype_code(xd), k, k, y.data_ptr(), nv.dtype_code(y), n, bd.data_ptr(), m, n, k, ws.data_ptr(),
                             ws.numel(), nv.stream_ptr(xd.device)), "pe_gemm")
        out.append(y)
    rows = torch.cat([torch.arange(0, m, 37), torch.arange(m - 3, m)])
    ref = oracle.linear_dequant(x[rows], codes, norms, cts) + bias.float()
    assert max_rel(out[0], out[1]) <= 1e-2 and max_rel(out[0][rows.cuda()], ref) <= TOL
    assert max_rel(out[0][rows.cuda()][:, -400:], ref[:, -400:]) <= TOL
    return out


@pytest.mark.parametrize("m,n,bits,dtype", [(300, 75 * 256 + 40, 4, torch.float16), (600, 37 * 256 + 101, 3, torch.float32),
                                            (1100, 25 * 256 + 8, 5, torch.bfloat16)])
def test_gemm_some_hundred_rows_with_and_without_room(m, n, bits, dtype):
    """Just over a wave of pair tiles: ragged edges, bias, every output type, whichever kernel and tiling either workspace leads to."""
    with_and_without_room(m, n, 4096, bits, dtype)


@pytest.mark.parametrize("m,n,bits,dtype", [(4097, 9 * 256 - 103, 4, torch.float32), (4300, 17 * 256 - 152, 3, torch.float16),
                                            (4150, 17 * 256 - 55, 6, torch.bfloat16), (4097, 25 * 256 - 200, 5, torch.float32)])
def test_gemm_last_wave_split_over_the_pairs(m, n, bits, dtype):
    """Waves of whole tiles and one column of tiles left, split in K: ragged edges in the split columns, partials that leave by TMA and
    that do not, bias, every output type.  The columns before them have the bits of the launch without room for the partials."""
    from polarengine_vllm_b200 import _native as nv
    k, split = 4096, (n - 1) // 256 * 256
    assert nv.lib().pe_gemm_workspace_bytes_splitk(m, n, k) >= nv.lib().pe_gemm_workspace_bytes(m, k) + 8 * m * (n - split) * 4
    room, none = with_and_without_room(m, n, k, bits, dtype)
    assert torch.equal(room[:, :split], none[:, :split]) and not torch.equal(room[:, split:], none[:, split:])


@pytest.mark.parametrize("m,n,k,bits", [(257, 100, 128, 4), (258, 4096, 1024, 3), (300, 1000, 640, 6), (385, 19000, 256, 4), (512, 2500, 2048, 5), (577, 130, 4096, 3),
                                        (640, 12300, 512, 4), (769, 2560, 384, 6), (1025, 1536, 1152, 4), (1600, 700, 896, 3), (1601, 700, 896, 3), (1537, 9000, 256, 5)])
def test_gemm_some_hundred_rows(m, n, k, bits):
    """257 rows and more: whichever kernel and tiling the estimate picks, with one or several tiles of rows, K ranges or none, ragged
    edges, a bias, 16- and 32-bit results, and a workspace without room for K ranges."""
    from polarengine_vllm_b200 import _native as nv, kernels, packing
    codes, norms, cts = rand_layer(n, k, bits, seed=m + n)
    packed, in_f = bits <= 4, k - 5
    w = packing.pack_codes_half_block(codes.cuda()) if packed else codes.cuda()
    nd, ctd, x, bias = norms.cuda(), cts.cuda(), rand_x(m, in_f, seed=k).cuda(), rand_x(1, n, seed=2)[0].cuda()
    ref = oracle.linear_dequant(x.cpu(), codes, norms, cts, in_f=in_f) + bias.cpu().float()
    for dt in (torch.float16, torch.float32):
        y = kernels.quant_matmul(w, packed, nd, ctd, x, False, n, in_f, k, dt, bias)
        assert y.dtype == dt and max_rel(y, ref) <= TOL
    lib, need = nv.lib(), nv.lib().pe_gemm_workspace_bytes(m, k)
    assert nv.lib().pe_gemm_workspace_bytes_splitk(m, n, k) >= need
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    y = torch.empty(m, n, device="cuda")
    nv.check(lib.pe_gemm(w.data_ptr(), int(packed), w.stride(0), nd.data_ptr(), nd.stride(0), ctd.data_ptr(), ctd.numel(), x.data_ptr(), nv.PE_X_RAW, nv.PE_F16,
                         x.stride(0), in_f, y.data_ptr(), nv.PE_F32, n, bias.data_ptr(), m, n, k, ws.data_ptr(), need, nv.stream_ptr(x.device)), "pe_gemm")
    assert max_rel(y, ref) <= TOL


@pytest.mark.parametrize("n,bits,dtype", [(19 * 256 + 40, 4, torch.float16), (18 * 256 + 256, 6, torch.float32), (700, 3, torch.bfloat16)])
def test_gemm_pairs_last_wave_split(n, bits, dtype):
    """Rows enough for pairs of CTAs whatever the estimate says: a last, partly filled wave cut into K ranges, and a launch of few tiles."""
    m, k = 4200, 2048
    codes, norms, cts = rand_layer(n, k, bits, seed=n)
    x = rand_x(m, k, seed=4)
    y = run_gemm(codes, norms, cts, x, bits, out_dtype=dtype)
    rows = torch.cat([torch.arange(0, m, 29), torch.arange(m - 20, m)])
    assert torch.isfinite(y.float()).all() and max_rel(y[rows.cuda()], oracle.linear_dequant(x[rows], codes, norms, cts)) <= TOL


@pytest.mark.parametrize("rows", [40, 300, 1700, 4200])
@pytest.mark.parametrize("bits", [4, 5])
def test_prefill_weights_rewritten_by_the_kernel_in_front(bits, rows):
    """Codes and norms rewritten on the device right before the call: the tensor-core kernels read them before their own wait, the
    preparation launch having waited for what wrote them."""
    from polarengine_vllm_b200 import kernels, packing
    n, k, sets = 1024, 1024, []
    for seed in (1, 2):
        codes, norms, ct = rand_layer(n, k, bits, seed=seed)
        sets.append((packing.pack_codes_half_block(codes.cuda()) if bits <= 4 else codes.cuda(), norms.cuda()))
    packed, ctd, x = bits <= 4, ct.cuda(), rand_x(rows, k, seed=3).cuda()
    want = [kernels.quant_matmul(w, packed, m, ctd, x, False, n, k, k, torch.float32) for w, m in sets]
    w, m = sets[0][0].clone(), sets[0][1].clone()
    kernels.quant_matmul(w, packed, m, ctd, x, False, n, k, k, torch.float32)
    graph, got = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph):
        for i in range(20):
            torch.add(sets[i % 2][0], 0, out=w)
            torch.mul(sets[i % 2][1], 1, out=m)
            got.append(kernels.quant_matmul(w, packed, m, ctd, x, False, n, k, k, torch.float32))
    graph.replay()
    assert all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))


@pytest.mark.parametrize("n,k,bits,few,many", [(4096, 4096, 6, 384, 512), (4096, 4096, 4, 387, 512), (4096, 12288, 4, 416, 512), (12288, 1024, 4, 400, 4200),
                                               (1536, 2048, 5, 257, 512), (300, 128, 3, 259, 5000), (2817, 640, 6, 511, 4700),
                                               (2560, 640, 5, 1700, 4200), (300, 1024, 4, 4096, 4097)])
def test_gemm_same_bits_where_k_is_cut_alike(n, k, bits, few, many):
    """The rows of a launch have the bits they have in a launch of more rows, whose larger number takes it to other tiles or to pairs of
    CTAs: where both cut K into the same ranges every product is added in the same order."""
    codes, norms, cts = rand_layer(n, k, bits, seed=n + k)
    x = rand_x(many, k, seed=few)
    a, b = run_gemm(codes, norms, cts, x[:few], bits, out_dtype=torch.float32), run_gemm(codes, norms, cts, x, bits, out_dtype=torch.float32)
    assert torch.equal(a, b[:few])
    ref = oracle.linear_dequant(x[:few], codes, norms, cts)
    assert max_rel(a, ref) <= TOL


@pytest.mark.parametrize("m,n,k,bits", [(1601, 1024, 8192, 3), (1700, 12288, 512, 4), (1700, 19 * 256 + 40, 2048, 6), (2050, 1000, 2176, 6), (2049, 2300, 5120, 4),
                                        (4096, 300, 1024, 5)])
def test_gemm_some_thousand_rows(m, n, k, bits):
    """1601 to 4096 rows on layers for which the estimate picks the tensor-memory kernel: many tiles of rows, one or two halves, K ranges
    or none, ragged edges, a bias, every output type."""
    codes, norms, cts = rand_layer(n, k, bits, seed=m + n)
    in_f = k - 5
    x, bias = rand_x(m, in_f, seed=k), rand_x(1, n, seed=2).reshape(n)
    rows = torch.cat([torch.arange(0, m, 41), torch.arange(m - 20, m)])
    ref = oracle.linear_dequant(x[rows], codes, norms, cts, in_f=in_f) + bias.float()
    for dt in (torch.float16, torch.float32, torch.bfloat16):
        y = run_gemm(codes, norms, cts, x, bits, out_dtype=dt, bias=bias, in_f=in_f)
        assert torch.isfinite(y.float()).all() and max_rel(y[rows.cuda()], ref) <= TOL
