"""Quantized MoE expert path against the oracle composition (softmax/top-k/renormalise,
silu(gate)*up, down, weighted sum; expert projections are quantized linears).  The
reference has no quantized MoE arithmetic, so this composition is pinned only through
its pieces."""
import pytest
import torch

import polar_oracle as oracle
from helpers import max_rel, rand_layer, rand_x

pytestmark = pytest.mark.gpu


def build(e, h, i, seed=0):
    from polarengine_vllm_b200.moe_method import PolarQuantMoEMethod
    g = torch.Generator().manual_seed(seed)
    method = PolarQuantMoEMethod(3, 4)
    layer = torch.nn.Module()
    method.create_weights(layer, e, h, i, torch.float16)
    layer = layer.cuda()
    experts = []
    for ex in range(e):
        q = {}
        for name, shape, bits in (("gate", (i, h), 3), ("up", (i, h), 3), ("down", (h, i), 4)):
            q[name] = oracle.quantize_tensor(torch.randn(*shape, generator=g) * 0.02, bits)
        method.load_expert(layer, ex, q["gate"], q["up"], q["down"])
        experts.append({n: (q[n]["codes"], q[n]["norms"], q[n]["ct_scaled"], None) for n in q})
    method.process_weights_after_loading(layer)
    return method, layer, experts


@pytest.mark.parametrize("tokens", [1, 5, 64, 200])
def test_moe_matches_oracle(tokens):
    e, h, i, top_k = 16, 384, 200, 4   # ragged intermediate: down-projection K pads 200 -> 256
    method, layer, experts = build(e, h, i)
    g = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, h, generator=g).half()
    gate_w = (torch.randn(e, h, generator=g) * 0.02).half()
    w, ids = oracle.moe_route(x, gate_w, top_k)
    ref = oracle.moe_forward(x, w, ids, experts)
    y = method.apply(layer, x.cuda(), w.cuda(), ids.cuda())
    assert y.shape == (tokens, h) and y.dtype == torch.float16
    assert max_rel(y, ref) <= 1e-2
    # the per-expert path (tensor-core kernel for experts with more than 16 rows) agrees
    y_loop = method._moe_forward_per_expert(layer, x.cuda(), w.cuda(), ids.cuda())
    assert max_rel(y_loop, ref) <= 1e-2
    # older contract: router logits in, routing done inside
    logits = (x.float() @ gate_w.float().T).cuda()
    y2 = method.apply(layer, x.cuda(), logits, top_k, True)
    assert max_rel(y2, ref) <= 1e-2


def test_moe_expert_parallel_partition_sums_to_full():
    e, h, i, top_k = 8, 256, 128, 2
    method, layer, experts = build(e, h, i, seed=3)
    g = torch.Generator().manual_seed(1)
    x = torch.randn(9, h, generator=g).half().cuda()
    w, ids = oracle.moe_route(x.cpu(), (torch.randn(e, h, generator=g) * 0.02).half(), top_k)
    full = method.moe_forward(layer, x, w.cuda(), ids.cuda()).float()
    parts = torch.zeros_like(full)
    for rank in range(2):
        emap = torch.full((e,), -1, dtype=torch.long)
        emap[rank * 4:(rank + 1) * 4] = torch.arange(4)
        sub = torch.nn.Module()
        for name in ("w13_codes", "w13_norms", "w2_codes", "w2_norms"):
            setattr(sub, name, getattr(layer, name)[rank * 4:(rank + 1) * 4])
        for name in ("w13_ct_scaled", "w2_ct_scaled", "moe_hidden", "moe_inter", "moe_hidden_padded", "moe_inter_padded"):
            setattr(sub, name, getattr(layer, name))
        parts += method.moe_forward(sub, x, w.cuda(), ids.cuda(), expert_map=emap.cuda()).float()
    assert max_rel(parts, full) <= 2e-3


def build_random_codes(e, h, i, seed=0):
    """Experts with uniformly random codes and |randn| norms (helpers.rand_layer): no quantizer run, so the
    128-expert layer of the benchmark configuration builds in seconds."""
    from helpers import rand_layer
    from polarengine_vllm_b200.moe_method import PolarQuantMoEMethod
    method = PolarQuantMoEMethod(3, 4)
    layer = torch.nn.Module()
    method.create_weights(layer, e, h, i, torch.float16)
    layer = layer.cuda()
    hp, ip = -(-h // 128) * 128, -(-i // 128) * 128
    experts = []
    for ex in range(e):
        q = {}
        for name, (n, kp, k), bits in (("gate", (i, hp, h), 3), ("up", (i, hp, h), 3), ("down", (h, ip, i), 4)):
            codes, norms, cts = rand_layer(n, kp, bits, seed=seed + 3 * ex + len(q))
            q[name] = {"codes": codes, "norms": norms, "ct_scaled": cts}
        method.load_expert(layer, ex, q["gate"], q["up"], q["down"])
        experts.append({n: (q[n]["codes"], q[n]["norms"], q[n]["ct_scaled"], None) for n in q})
    method.process_weights_after_loading(layer)
    return method, layer, experts


@pytest.mark.parametrize("tokens", [1, 64, 2048])
def test_moe_benchmark_configuration(tokens):
    """128 experts, top-8, hidden 2688, intermediate 1856 (down-projection K pads to 1920): the shapes of the
    expert-layer benchmark.  64 tokens run the decode-size grouped launches (pe_gemv_grouped), 2048 the
    grouped tensor-core launches (pe_gemm_grouped, about 2000 device-built tiles).  The GPU computes every
    token; the CPU oracle (routing, silu(gate)*up, down, weighted sum: nemotron_offload.py:180-226) is
    evaluated on a sample of them."""
    e, h, i, top_k = 128, 2688, 1856, 8
    method, layer, experts = build_random_codes(e, h, i, seed=500)
    g = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, h, generator=g).half()
    gate_w = (torch.randn(e, h, generator=g) * 0.02).half()
    w, ids = oracle.moe_route(x, gate_w, top_k)
    y = method.apply(layer, x.cuda(), w.cuda(), ids.cuda())
    assert y.shape == (tokens, h) and y.dtype == torch.float16 and torch.isfinite(y.float()).all()
    sample = torch.arange(tokens) if tokens <= 64 else torch.randperm(tokens, generator=g)[:24].sort().values
    ref = oracle.moe_forward(x[sample], w[sample], ids[sample], experts)
    assert max_rel(y[sample.cuda()], ref) <= 1e-2


@pytest.mark.parametrize("t,e,k", [(1, 128, 8), (64, 128, 8), (300, 60, 4), (7, 1000, 32)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_routing_kernel_matches_softmax_topk(t, e, k, dtype):
    """pe_moe_route = softmax (fp32) -> top-k -> renormalise of nemotron_offload.py:180-189: the same weights as
    torch.topk on the same logits to fp32 rounding (and the same experts in the same order where no two logits are
    equal); with and without renormalisation."""
    from polarengine_vllm_b200.moe_method import route_softmax_topk
    g = torch.Generator().manual_seed(t + e)
    logits = (torch.randn(t, e, generator=g) * 3).to(dtype)
    for renorm in (True, False):
        w, ids = route_softmax_topk(logits.cuda(), k, renorm)
        p = torch.softmax(logits.float(), dim=-1)
        rw, rids = p.topk(k, dim=-1)
        if renorm:
            rw = rw / rw.sum(-1, keepdim=True)
        assert ids.dtype == torch.int64 and w.dtype == torch.float32
        w, ids = w.cpu(), ids.cpu()
        # the k largest probabilities in descending order (equal logits -- common in 16-bit -- may swap places or, at
        # the k-th place, experts: either choice is a valid top-k), each weight being its own expert's probability
        assert torch.allclose(w, rw, rtol=1e-5, atol=1e-7)
        own = p.gather(1, ids)
        if renorm:
            own = own / own.sum(-1, keepdim=True)
        assert torch.allclose(w, own, rtol=1e-5, atol=1e-7)
        assert all(len(set(r.tolist())) == k for r in ids)
        if dtype == torch.float32:
            assert torch.equal(ids, rids)


@pytest.mark.parametrize("t,e,k,mapped", [(1, 128, 8, False), (32, 60, 32, False), (33, 256, 4, True), (7, 1000, 3, True)])
def test_joint_routing_and_plan_equals_the_two_launches(t, e, k, mapped):
    """pe_moe_route_plan against pe_moe_route followed by a plan made on the host: the same weights and ids, every
    pair's row inside its expert's range, and problems that cover the rows of each expert in pieces of eight."""
    from polarengine_vllm_b200 import _native as nv
    from polarengine_vllm_b200.moe_method import route_softmax_topk
    g = torch.Generator().manual_seed(t * e)
    logits = torch.randn(t, e, generator=g).cuda()
    local = (e + 1) // 2 if mapped else e
    emap = torch.where(torch.arange(e) % 2 == 0, torch.arange(e) // 2, -1) if mapped else torch.arange(e)
    demap, pairs, cap = emap.cuda(), t * k, min(local, t * k) + t * k // 8
    w, ids = torch.empty(t, k, device="cuda"), torch.empty(t, k, dtype=torch.int64, device="cuda")
    tok, pos = (torch.full((pairs,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    prob, rows = torch.empty(cap, 4, dtype=torch.int32, device="cuda"), torch.empty(local, 2, dtype=torch.int32, device="cuda")
    nv.check(nv.lib().pe_moe_route_plan(logits.data_ptr(), 0, e, t, e, k, 1, w.data_ptr(), ids.data_ptr(), demap.data_ptr() if mapped else None,
                                        e if mapped else 0, local, 8, cap, tok.data_ptr(), pos.data_ptr(), prob.data_ptr(), rows.data_ptr(),
                                        nv.stream_ptr(logits.device)), "pe_moe_route_plan")
    rw, rids = route_softmax_topk(logits, k, True)
    assert torch.equal(w, rw) and torch.equal(ids, rids)
    own = emap[ids.cpu()].flatten()
    count = torch.bincount(own[own >= 0], minlength=local)
    assert torch.equal(rows.cpu()[:, 1].long(), count) and torch.equal(rows.cpu()[:, 0].long(), count.cumsum(0) - count)
    p, first = pos.cpu().long(), rows.cpu()[:, 0].long()
    assert torch.equal(p < 0, own < 0)
    live = own >= 0
    assert (p[live] >= first[own[live]]).all() and (p[live] < (first + count)[own[live]]).all() and p[live].unique().numel() == int(live.sum())
    assert torch.equal(tok.cpu().long()[p[live]], torch.arange(pairs)[live] // k)
    want = [(x, int(first[x]) + 8 * j, min(8, int(count[x]) - 8 * j)) for x in range(local) for j in range(-(-int(count[x]) // 8))]
    got = [tuple(r[:3]) for r in prob.cpu().tolist()]
    assert got[:len(want)] == want and all(r[2] == 0 for r in got[len(want):])


@pytest.mark.parametrize("bits", [3, 4, 5])
@pytest.mark.parametrize("counts", [(0, 1, 15, 16, 17, 0), (96, 97, 128, 129, 0, 3), (192, 193, 384, 385, 0, 0)])
def test_grouped_tensor_core_launch_edges(counts, bits):
    """pe_gemm_grouped and pe_gemm_grouped_silu_mul at the edges of their tiles: empty experts, token counts around 16,
    around the 96 where a tile's accumulators stop alternating, and around 192 where an expert takes two; out columns
    that are not whole tiles; rows taken by index, and rows sent to theirs."""
    from polarengine_vllm_b200 import _native as nv, packing
    n, k, in_f, e, rows, tokens = 2 * 200, 384, 300, len(counts), sum(counts), 64
    dev, packed = torch.device("cuda"), bits <= 4
    nv.ensure_init(dev)
    lib = nv.lib()
    ws_bytes = lib.pe_gemm_grouped_workspace_bytes(e, rows, n, k)
    layers = [rand_layer(n, k, bits, seed=bits + i) for i in range(e)]
    codes = torch.stack([packing.pack_codes_half_block(c.cuda()) if packed else c.cuda() for c, _, _ in layers])
    norms, ct = torch.stack([m for _, m, _ in layers]).cuda(), layers[0][2].cuda()
    first = torch.tensor(counts).cumsum(0) - torch.tensor(counts)
    spans = torch.stack([first, torch.tensor(counts)], 1).int().cuda()
    x, pick = rand_x(tokens, in_f, seed=1), torch.randint(0, tokens, (rows,), generator=torch.Generator().manual_seed(2))
    pd, xd, ws = pick.int().cuda(), x.cuda(), torch.empty(ws_bytes, dtype=torch.uint8, device=dev)
    y = torch.full((rows, n), float("nan"), device=dev)
    act = torch.full((rows, n // 2), float("nan"), dtype=torch.float16, device=dev)
    # the list as scattered rows of another order: row i of `xs` is row to[i] of the list
    to = torch.randperm(rows, generator=torch.Generator().manual_seed(3))
    xs, td = x[pick][to].contiguous().cuda(), to.int().cuda()
    head = (codes.data_ptr(), int(packed), codes.stride(1), codes.stride(0), norms.data_ptr(), norms.stride(1), norms.stride(0), ct.data_ptr(),
            ct.numel())
    raw = (nv.PE_X_RAW, nv.dtype_code(xd), xd.stride(0), in_f)
    tail = (spans.data_ptr(), e, rows, n, k, ws.data_ptr(), ws.numel(), nv.stream_ptr(dev))
    nv.check(lib.pe_gemm_grouped(*head, xd.data_ptr(), *raw, pd.data_ptr(), y.data_ptr(), nv.PE_F32, n, *tail), "pe_gemm_grouped")
    nv.check(lib.pe_gemm_grouped_silu_mul(*head, xs.data_ptr(), *raw, td.data_ptr(), rows, 1, act.data_ptr(), n // 2, *tail), "pe_gemm_grouped_silu_mul")
    assert int(ws[:4].view(torch.int32)) == 0
    xr = x[pick]
    ref = torch.cat([oracle.linear_dequant(xr[int(first[i]):int(first[i]) + c], *layers[i], in_f=in_f) for i, c in enumerate(counts) if c])
    assert max_rel(y, ref) <= 1e-2
    assert max_rel(act, torch.nn.functional.silu(ref[:, :n // 2]) * ref[:, n // 2:]) <= 1e-2


@pytest.mark.parametrize("bits,inter,h", [(4, 296, 257), (5, 1920, 144)])
def test_grouped_tiled_silu_input_equals_row_major(bits, inter, h):
    """pe_gemv_grouped_tiled = pe_gemv_grouped bit for bit, with silu(gate) * up computed where the input is prepared equal
    to the activation launch in front (ragged widths, problems of 0, 1, 8, 9 and 16 rows)."""
    from polarengine_vllm_b200 import _native as nv, kernels, packing
    from polarengine_vllm_b200.decode_ops import silu_mul
    sizes, kp, dev, packed = (1, 8, 0, 9, 16), -(-inter // 128) * 128, torch.device("cuda"), bits <= 4
    nv.ensure_init(dev)
    lib = nv.lib()
    layers = [rand_layer(h, kp, bits, seed=i) for i in range(len(sizes))]
    codes = torch.stack([packing.pack_codes_half_block(c.cuda()) if packed else c.cuda() for c, _, _ in layers])
    norms, ct = torch.stack([m for _, m, _ in layers]).cuda(), layers[0][2].cuda()
    tiles = torch.cat([kernels.retile(codes[i], packed, norms[i]) for i in range(len(sizes))])
    rows = sum(sizes)
    first = [sum(sizes[:i]) for i in range(len(sizes))]
    prob = torch.tensor([[i, first[i], s, 0] for i, s in enumerate(sizes)], dtype=torch.int32).cuda()
    gu = rand_x(rows, 2 * inter, seed=3).cuda()
    act = silu_mul(gu, inter)
    ws = nv.grouped_scratch(dev, lib.pe_gemv_grouped_workspace_bytes(len(sizes), h, kp))
    out = []
    for x, kind in ((act, nv.PE_X_RAW), (gu, nv.PE_X_SILU_MUL)):
        args = (ct.data_ptr(), ct.numel(), x.data_ptr(), kind, nv.dtype_code(x), x.stride(0), inter, None)
        for tiled in (False, True):
            y = torch.zeros(rows, h, device=dev)
            end = (y.data_ptr(), nv.PE_F32, h, prob.data_ptr(), len(sizes), 16, h, kp, ws.data_ptr(), ws.numel(), nv.stream_ptr(dev))
            if tiled:
                nv.check(lib.pe_gemv_grouped_tiled(tiles.data_ptr(), int(packed), tiles.numel() // len(sizes), *args, *end), "tiled")
            else:
                nv.check(lib.pe_gemv_grouped(codes.data_ptr(), int(packed), codes.stride(1), codes.stride(0), norms.data_ptr(), norms.stride(1),
                                             norms.stride(0), *args, *end), "row-major")
            out.append(y)
    assert all(torch.equal(out[0], y) for y in out[1:])
    a = act.cpu()
    ref = torch.cat([oracle.linear_dequant(a[first[i]:first[i] + s], *layers[i], in_f=inter) for i, s in enumerate(sizes) if s])
    assert max_rel(out[0], ref) <= 1e-2


@pytest.mark.parametrize("tokens", [1, 6])
def test_experts_have_one_copy_of_their_weights(tokens):
    """Decode-size batches multiply by what the experts' arrays hold at the call -- rewritten in place included, the first
    call inside a capture included -- and leave no further memory with the layer."""
    e, h, i, top_k = 16, 640, 384, 4
    method, layer, _ = build_random_codes(e, h, i, seed=1)
    _, other, experts = build_random_codes(e, h, i, seed=7)
    g = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, h, generator=g).half()
    w, ids = oracle.moe_route(x, (torch.randn(e, h, generator=g) * 0.02).half(), top_k)
    xd, wd, idd = x.cuda(), w.cuda(), ids.cuda()
    want = method.apply(other, xd, wd, idd)
    assert max_rel(want, oracle.moe_forward(x, w, ids, experts)) <= 1e-2
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held = method.apply(layer, xd, wd, idd)  # the layer's first call
    graph.replay()
    y = method.apply(layer, xd, wd, idd)
    assert torch.equal(y, held)
    for name in ("w13_codes", "w13_norms", "w2_codes", "w2_norms"):
        getattr(layer, name).data.copy_(getattr(other, name).data)
    assert torch.equal(method.apply(layer, xd, wd, idd), want)
    graph.replay()
    assert torch.equal(held, want)
    assert not [k for k, v in vars(layer).items() if torch.is_tensor(v)]  # parameters and buffers only


@pytest.mark.parametrize("rows,kp,bits", [(257, 384, 4), (40, 1024, 3), (33, 1152, 5), (16, 4224, 4), (8, 640, 6)])
def test_grouped_norms_however_they_lie(rows, kp, bits):
    """pe_gemv_grouped with the norms of a tile in one piece (a last tile whose norms are not whole 16 bytes, or two K
    ranges, excepted) and with a gap between rows, between experts, or at an odd address: the same bits, and the oracle's
    values."""
    from polarengine_vllm_b200 import _native as nv, packing
    sizes, dev, packed = (3, 0, 8), torch.device("cuda"), bits <= 4
    nv.ensure_init(dev)
    lib, nb = nv.lib(), kp // 128
    layers = [rand_layer(rows, kp, bits, seed=i) for i in range(len(sizes))]
    codes = torch.stack([packing.pack_codes_half_block(c.cuda()) if packed else c.cuda() for c, _, _ in layers])
    dense, ct = torch.stack([m for _, m, _ in layers]).cuda(), layers[0][2].cuda()
    first, total = [0, 3, 3], sum(sizes)
    prob = torch.tensor([[i, first[i], s, 0] for i, s in enumerate(sizes)], dtype=torch.int32).cuda()
    x = rand_x(total, kp, seed=3).cuda()
    ws = nv.grouped_scratch(dev, lib.pe_gemv_grouped_workspace_bytes(len(sizes), rows, kp))
    out = []
    for gap_row, gap_expert, shift in ((0, 0, 0), (1, 0, 0), (0, 3, 0), (0, 0, 1)):
        buf = torch.full((len(sizes) * (rows * (nb + gap_row) + gap_expert) + 8,), float("nan"), dtype=torch.float16, device=dev)
        m = torch.as_strided(buf, (len(sizes), rows, nb), (rows * (nb + gap_row) + gap_expert, nb + gap_row, 1), shift)
        m.copy_(dense)
        y = torch.zeros(total, rows, device=dev)
        nv.check(lib.pe_gemv_grouped(codes.data_ptr(), int(packed), codes.stride(1), codes.stride(0), m.data_ptr(), m.stride(1), m.stride(0),
                                     ct.data_ptr(), ct.numel(), x.data_ptr(), nv.PE_X_RAW, nv.dtype_code(x), x.stride(0), kp, None, y.data_ptr(),
                                     nv.PE_F32, rows, prob.data_ptr(), len(sizes), 8, rows, kp, ws.data_ptr(), ws.numel(), nv.stream_ptr(dev)),
                 "pe_gemv_grouped")
        out.append(y)
    ref = torch.cat([oracle.linear_dequant(x.cpu()[first[i]:first[i] + s], *layers[i]) for i, s in enumerate(sizes) if s])
    assert max_rel(out[0], ref) <= 1e-2
    assert all(torch.equal(out[0], y) for y in out[1:])


@pytest.mark.parametrize("rows,kp,bits", [(2100, 2688, 3), (1000, 2176, 6), (300, 128, 4)])
def test_grouped_norms_gathered_over_several_passes(rows, kp, bits):
    """Rows of up to 21 blocks whose norms have gaps, more tiles of rows than SMs: gathered by a warp of their own, the bits of
    copied norms.  Problems of every size, an empty one and more of them than are used."""
    from polarengine_vllm_b200 import _native as nv, packing
    sizes, dev, packed, nb = (8, 1, 0, 5, 7), torch.device("cuda"), bits <= 4, kp // 128
    nv.ensure_init(dev)
    lib = nv.lib()
    layers = [rand_layer(rows, kp, bits, seed=i) for i in range(len(sizes))]
    codes = torch.stack([packing.pack_codes_half_block(c.cuda()) if packed else c.cuda() for c, _, _ in layers])
    dense, ct = torch.stack([m for _, m, _ in layers]).cuda(), layers[0][2].cuda()
    gaps = torch.full((len(sizes), rows, nb + 3), float("nan"), dtype=torch.float16, device=dev)
    gaps[:, :, 1:1 + nb] = dense
    first = [sum(sizes[:i]) for i in range(len(sizes))]
    prob = torch.tensor([[i, first[i], s, 0] for i, s in enumerate(sizes)] + [[0, 0, 0, 0]] * 3, dtype=torch.int32).cuda()
    x = rand_x(sum(sizes), kp, seed=3).cuda()
    ws = nv.grouped_scratch(dev, lib.pe_gemv_grouped_workspace_bytes(len(prob), rows, kp))
    out = []
    for m in (dense, gaps[:, :, 1:1 + nb]):
        y = torch.full((sum(sizes), rows), float("nan"), device=dev)
        nv.check(lib.pe_gemv_grouped(codes.data_ptr(), int(packed), codes.stride(1), codes.stride(0), m.data_ptr(), m.stride(1), m.stride(0),
                                     ct.data_ptr(), ct.numel(), x.data_ptr(), nv.PE_X_RAW, nv.dtype_code(x), x.stride(0), kp, None, y.data_ptr(),
                                     nv.PE_F32, rows, prob.data_ptr(), len(prob), 8, rows, kp, ws.data_ptr(), ws.numel(), nv.stream_ptr(dev)),
                 "pe_gemv_grouped")
        out.append(y)
    ref = torch.cat([oracle.linear_dequant(x.cpu()[first[i]:first[i] + s], *layers[i]) for i, s in enumerate(sizes) if s])
    assert max_rel(out[0], ref) <= 1e-2 and torch.equal(out[0], out[1])


@pytest.mark.parametrize("max_rows,rows,kp,bits", [(16, 3000, 2176, 4), (16, 1500, 4224, 3), (16, 1501, 2048, 5), (16, 1200, 2560, 6), (16, 3000, 1024, 4),
                                                   (8, 3000, 2560, 6), (8, 1500, 4096, 4), (8, 700, 4096, 5)])
def test_grouped_rings_and_sets_of_sums(max_rows, rows, kp, bits):
    """Problems of 8 and 16 rows over several passes a CTA, with one set of partial sums and with two, passes of 32, 64 and 128 rows, one
    and several chunks of K: the oracle's values, the bits of the tiled copy, and the same bits every time."""
    from polarengine_vllm_b200 import _native as nv, kernels, packing
    sizes, dev, packed = (max_rows, 1, 0, 7, max_rows, 3), torch.device("cuda"), bits <= 4
    nv.ensure_init(dev)
    lib = nv.lib()
    layers = [rand_layer(rows, kp, bits, seed=i) for i in range(len(sizes))]
    codes = torch.stack([packing.pack_codes_half_block(c.cuda()) if packed else c.cuda() for c, _, _ in layers])
    norms, ct = torch.stack([m for _, m, _ in layers]).cuda(), layers[0][2].cuda()
    tiles = torch.cat([kernels.retile(codes[i], packed, norms[i]) for i in range(len(sizes))])
    first = [sum(sizes[:i]) for i in range(len(sizes))]
    prob = torch.tensor([[i, first[i], s, 0] for i, s in enumerate(sizes)], dtype=torch.int32).cuda()
    x = rand_x(sum(sizes), kp, seed=3).cuda()
    ws = nv.grouped_scratch(dev, lib.pe_gemv_grouped_workspace_bytes(len(sizes), rows, kp))
    tail = (prob.data_ptr(), len(sizes), max_rows, rows, kp, ws.data_ptr(), ws.numel(), nv.stream_ptr(dev))
    out = []
    for tiled in (False, False, True):
        y = torch.full((sum(sizes), rows), float("nan"), device=dev)
        mid = (ct.data_ptr(), ct.numel(), x.data_ptr(), nv.PE_X_RAW, nv.dtype_code(x), x.stride(0), kp, None, y.data_ptr(), nv.PE_F32, rows)
        if tiled:
            nv.check(lib.pe_gemv_grouped_tiled(tiles.data_ptr(), int(packed), tiles.numel() // len(sizes), *mid, *tail), "tiled")
        else:
            nv.check(lib.pe_gemv_grouped(codes.data_ptr(), int(packed), codes.stride(1), codes.stride(0), norms.data_ptr(), norms.stride(1),
                                         norms.stride(0), *mid, *tail), "row-major")
        out.append(y)
    ref = torch.cat([oracle.linear_dequant(x.cpu()[first[i]:first[i] + s], *layers[i]) for i, s in enumerate(sizes) if s])
    assert max_rel(out[0], ref) <= 1e-2 and torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
