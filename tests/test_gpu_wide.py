"""GPU parity tests of the wide (prefill) MoE path: expert-major permute, grouped dequant GEMM on
tcgen05/TMEM, SwiGLU, rank-ordered unpermute. Same oracle, same tolerances as the narrow path:
identical expert selection, relative L2 <= 1e-3 against the CPU path. The reference's own op table
stops at 62 rows (src/graph/worklist.c:316); per-token semantics are the CPU path's, so parity is
checked token by token."""
import numpy as np
import pytest

from golden_cases import CASES, layer_inputs
from yvex_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from yvex_b200 import lib
    return lib


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def run_layer(L, spec, weights, router, x, logits, wide=True):
    t = {k: dev(v.reshape(-1)) for k, v in weights.items()}
    if router is not None:
        t["router"] = dev(router)
    st = L.Status()
    out, sel, w = L.moe_layer(L.geometry_of(spec), L.weights_of(t), dev(x), st,
                              logits=None if logits is None else dev(logits), wide=wide)
    return out.cpu().numpy(), sel.cpu().numpy(), w.cpu().numpy(), st.read()


@pytest.mark.parametrize("name", list(CASES["layer"]))
def test_wide_layer_vs_frozen_reference(L, golden, name):
    spec, weights, router, x, logits = layer_inputs(name)           # IQ2_XXS gate/up, Q2_K down
    out, sel, w, status = run_layer(L, spec, weights, router, x, logits)
    assert status == 0
    assert (sel == golden[f"layer_{name}_sel"]).all()
    want = golden[f"layer_{name}_out"].view(np.float32)
    assert rel_l2(out, want) <= 1e-3, rel_l2(out, want)
    assert (synth.bf16_round(out).view(np.uint32) == out.view(np.uint32)).all()


@pytest.mark.parametrize("down", [synth.Q4_K, synth.Q2_K, synth.IQ2_XXS])
def test_wide_layer_ragged_groups_vs_oracle(L, port, down):
    """300 tokens over 8 experts: groups larger than one 128-column tile, ragged tails, and the
    shared expert's 3 token blocks. Q4_K is checked against this repository's restatement
    (reference-unpinned), the others against the reference-pinned port."""
    H, E, k, I, T = 512, 8, 2, 512, 300
    spec = synth.MoELayerSpec(H, E, k, I, down_qtype=down)
    rng = np.random.default_rng(41 + down)
    x = rng.standard_normal((T, H)).astype(np.float32)
    logits = rng.standard_normal((T, E)).astype(np.float32)
    logits[:, 5] -= 50.0                                   # expert 5 receives no token: empty group
    weights = synth.moe_weights(spec, 40 + down)
    Lp = port.layer(spec, weights, allow_q4k=True)
    rc, want, sel0, w0 = port.moe_tokens(Lp, x, logits=logits, threads=8)
    out, sel, w, status = run_layer(L, spec, weights, None, x, logits)
    assert rc == 0 and status == 0 and (sel == sel0).all() and not (sel == 5).any()
    assert rel_l2(out, want) <= 1e-3, rel_l2(out, want)
    per_token = np.linalg.norm(out - want, axis=1) / np.linalg.norm(want, axis=1)
    assert per_token.max() <= 4e-3, per_token.max()


@pytest.mark.parametrize("gate", [synth.Q2_K, synth.Q4_K])
def test_wide_layer_affine_gate_and_up_vs_oracle(L, port, gate):
    """Gate and up weights of a qtype with a min term: the fused gate/up GEMM then needs the sub-block
    sums of the ACTIVATION rows as its second operand. 300 tokens over 8 experts, ragged groups."""
    H, E, k, I, T = 512, 8, 2, 256, 300
    spec = synth.MoELayerSpec(H, E, k, I, gate_qtype=gate, down_qtype=synth.IQ2_XXS)
    rng = np.random.default_rng(70 + gate)
    x = rng.standard_normal((T, H)).astype(np.float32)
    logits = rng.standard_normal((T, E)).astype(np.float32)
    weights = synth.moe_weights(spec, 71 + gate)
    Lp = port.layer(spec, weights, allow_q4k=True)
    rc, want, sel0, w0 = port.moe_tokens(Lp, x, logits=logits, threads=8)
    out, sel, w, status = run_layer(L, spec, weights, None, x, logits)
    assert rc == 0 and status == 0 and (sel == sel0).all()
    assert rel_l2(out, want) <= 1e-3, rel_l2(out, want)


def test_expert_parallel_building_blocks_match_single_device_layer_bit_for_bit(L):
    """The expert-parallel decomposition (route -> per-pair rows on the expert shard -> combine on
    the home rank), run here on one rank that owns every expert, and again with the experts split
    into two shards executed one after the other, must equal the fused wide layer exactly: pairs
    travel as whole bf16 rows and are summed in rank order."""
    import torch
    from yvex_b200.ep import DeviceOps, ExpertParallelLayer
    H, E, k, I, T = 512, 8, 2, 256, 200
    spec = synth.MoELayerSpec(H, E, k, I, down_qtype=synth.Q4_K)
    rng = np.random.default_rng(5)
    x, logits = dev(rng.standard_normal((T, H)).astype(np.float32)), dev(rng.standard_normal((T, E)).astype(np.float32))
    t = {kk: dev(v.reshape(-1)) for kk, v in synth.moe_weights(spec, 9).items()}
    st = L.Status()
    g, w = L.geometry_of(spec), L.weights_of(t)
    want, sel0, _ = L.moe_layer(g, w, x, st, logits=logits, wide=True)
    layer = ExpertParallelLayer(E, k, DeviceOps(g, g, w, st))
    got, sel, _ = layer.forward(x, logits)
    assert st.read() == 0 and torch.equal(sel, sel0)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    # two shards of 4 experts, pairs routed to each by hand
    xh = x.to(torch.bfloat16).to(torch.float16)
    sel, wts, _ = L.moe_route(g, w, st, logits=logits)
    y = torch.empty((T * k, H), dtype=torch.bfloat16, device="cuda")
    half = synth.MoELayerSpec(H, E // 2, k, I, down_qtype=synth.Q4_K)
    for shard in range(2):
        ts = dict(t)
        for name in ("gate", "up", "down"):
            per = t[name].numel() // E
            ts[name] = t[name][shard * 4 * per:(shard + 1) * 4 * per]
        mask = (sel.reshape(-1) // 4) == shard
        idx = mask.nonzero().reshape(-1)
        rows = xh.index_select(0, idx // k)
        y[idx] = L.moe_expert_rows(L.geometry_of(half), L.weights_of(ts), rows, (sel.reshape(-1)[idx] % 4).contiguous(),
                                   wts.reshape(-1)[idx].contiguous(), st)
    ysh = L.moe_expert_rows(g, w, xh, torch.full((T,), -1, dtype=torch.int32, device="cuda"),
                            torch.ones(T, device="cuda"), st)
    out2 = L.moe_combine(y, ysh, k, st)
    assert st.read() == 0 and torch.equal(out2.view(torch.int32), want.view(torch.int32))


def test_rows_stored_by_address_and_bad_trailers_are_dropped(L):
    """The down GEMM's epilogue stores every pair's row at home_bases[home rank] + home pair * hidden * 2 (here both
    "ranks" are buffers of this device): equal to the rows the list-order entry returns; a trailer that names a rank or
    a pair out of range sets status 2 and leaves its row unwritten."""
    import torch
    H, E, k, I, T = 512, 8, 2, 256, 150
    spec = synth.MoELayerSpec(H, E, k, I, down_qtype=synth.Q2_K)
    rng = np.random.default_rng(77)
    x, logits = dev(rng.standard_normal((T, H)).astype(np.float32)), dev(rng.standard_normal((T, E)).astype(np.float32))
    t = {kk: dev(v.reshape(-1)) for kk, v in synth.moe_weights(spec, 78).items()}
    st = L.Status()
    g, w = L.geometry_of(spec), L.weights_of(t)
    xh = x.to(torch.bfloat16).to(torch.float16)
    sel, wts, _ = L.moe_route(g, w, st, logits=logits)
    payload, inverse, counts = L.ep_dispatch_payload(xh, sel, wts, E, 1, 1, st, rank=0)
    want = L.moe_expert_rows_payload(g, w, payload, st)                     # rows in payload order
    home = torch.zeros((2, T * k, H), dtype=torch.bfloat16, device="cuda")
    bases = torch.tensor([home[0].data_ptr(), home[1].data_ptr()], dtype=torch.int64, device="cuda")
    trailers = payload[:, 2 * H:].view(torch.int32)                        # {local expert, weight, home pair, home rank}
    trailers[::2, 3] = 1                                                    # every other pair lives on "rank" 1
    L.moe_expert_rows_scatter(g, w, payload, bases, T * k, st)
    torch.cuda.synchronize()
    assert st.read() == 0
    pair = trailers[:, 2].long()
    rank = trailers[:, 3].long()
    got = home[rank, pair]
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert int((home.view(torch.int16) != 0).any(dim=2).sum()) == T * k    # nothing stored anywhere else
    home.zero_()
    trailers[0, 3] = 2                                                      # no such rank
    trailers[1, 2] = T * k                                                  # no such pair
    L.moe_expert_rows_scatter(g, w, payload, bases, T * k, st)
    torch.cuda.synchronize()
    assert st.read() == 2
    assert int((home.view(torch.int16) != 0).any(dim=2).sum()) == T * k - 2


def tokens_covering_all_experts(sel, count):
    """Indices of `count` rows of `sel` [T, k] chosen greedily so that every expert is selected by at least one."""
    sel = np.asarray(sel)
    need = set(np.unique(sel).tolist())
    picked = []
    for t in range(sel.shape[0]):
        hit = need.intersection(sel[t].tolist())
        if hit:
            picked.append(t)
            need -= hit
        if not need:
            break
    rest = [t for t in range(sel.shape[0] - 1, -1, -1) if t not in set(picked)]
    picked += rest[:max(0, count - len(picked))]
    return np.array(sorted(picked[:max(count, len(picked))]), np.int64)


def test_wide_matches_narrow_path_at_prefill_size(L, port):
    """Config-3 geometry (2048 tokens, hidden 4096, 64 experts top-6, inter 1536, IQ2_XXS + Q4_K):
    a sample of rows must agree with the narrow path run on those rows alone (rows are
    independent), and 64 rows that between them route to every one of the 64 experts must agree
    with the CPU path (each expert's weight offsets and tile positions are then exercised)."""
    import os
    import torch
    from yvex_b200.workloads import MoEWorkload
    wl = MoEWorkload("c3", 3)
    x, logits = wl.tokens(2048)
    st = L.Status()
    g, w = L.geometry_of(wl.spec), L.weights_of(wl.tensors)
    out, sel, wt = L.moe_layer(g, w, x, st, logits=logits, wide=True)
    idx = torch.tensor([0, 1, 127, 128, 777, 1500, 2046, 2047], device="cuda")
    out_n, sel_n, _ = L.moe_layer(g, w, x[idx].contiguous(), st, logits=logits[idx].contiguous(), wide=False)
    assert st.read() == 0 and (sel[idx] == sel_n).all()
    assert rel_l2(out[idx].cpu().numpy(), out_n.cpu().numpy()) <= 5e-4
    hw, _ = wl.host_copy()
    Lp = port.layer(wl.spec, hw, allow_q4k=True)
    pick = tokens_covering_all_experts(sel.cpu().numpy(), 64)
    assert pick.size >= 64 and set(np.unique(sel.cpu().numpy()[pick]).tolist()) == set(range(64))
    tp = torch.from_numpy(pick).cuda()
    rc, want, sel0, _ = port.moe_tokens(Lp, x[tp].cpu().numpy(), logits=logits[tp].cpu().numpy(), threads=os.cpu_count() or 8)
    assert rc == 0 and (sel[tp].cpu().numpy() == sel0).all()
    got = out[tp].cpu().numpy()
    assert rel_l2(got, want) <= 1e-3
    per_token = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert per_token.max() <= 4e-3, per_token.max()


def test_wide_config3_pinned_twin_vs_oracle(L, port):
    """The same geometry with Q2_K down weights - the qtype the reference's own MoE path decodes - so
    that the prefill path has a reference-pinned check at full size, on 64 rows covering all experts."""
    import os
    import torch
    from yvex_b200.workloads import MoEWorkload
    wl = MoEWorkload("c3", 3, down_qtype=synth.Q2_K)
    x, logits = wl.tokens(2048)
    st = L.Status()
    out, sel, _ = L.moe_layer(L.geometry_of(wl.spec), L.weights_of(wl.tensors), x, st, logits=logits, wide=True)
    hw, _ = wl.host_copy()
    Lp = port.layer(wl.spec, hw)
    pick = tokens_covering_all_experts(sel.cpu().numpy(), 64)
    tp = torch.from_numpy(pick).cuda()
    rc, want, sel0, _ = port.moe_tokens(Lp, x[tp].cpu().numpy(), logits=logits[tp].cpu().numpy(), threads=os.cpu_count() or 8)
    assert rc == 0 and st.read() == 0 and (sel[tp].cpu().numpy() == sel0).all()
    assert rel_l2(out[tp].cpu().numpy(), want) <= 1e-3


def test_wide_config5_size_properties(L, port):
    """Config-5 geometry on one device (16 384 tokens, hidden 7168, 256 experts top-8 + shared, inter 2048,
    IQ2_XXS + Q4_K). Size-independent properties: rows are independent, so a permuted batch gives the
    permuted result bit for bit (other column blocks, other tiles, same per-row arithmetic) and a
    sample of rows agrees with the decode path run on those rows alone; 16 rows spread over the batch
    are checked against the CPU path within the layer tolerance."""
    import os
    import torch
    from yvex_b200.workloads import MoEWorkload
    wl = MoEWorkload("c5", 5)
    T = wl.cfg["tokens"]
    x, logits = wl.tokens(T)
    st = L.Status()
    g, w = L.geometry_of(wl.spec), L.weights_of(wl.tensors)
    ws = torch.empty(L.moe_workspace_bytes(g, T, True), dtype=torch.uint8, device="cuda")
    out, sel, wt = L.moe_layer(g, w, x, st, logits=logits, wide=True, workspace=ws)
    assert st.read() == 0 and torch.isfinite(out).all()
    perm = torch.randperm(T, device="cuda", generator=torch.Generator(device="cuda").manual_seed(11))
    out_p, sel_p, _ = L.moe_layer(g, w, x[perm].contiguous(), st, logits=logits[perm].contiguous(), wide=True, workspace=ws)
    assert st.read() == 0 and (sel_p == sel[perm]).all()
    assert torch.equal(out_p.view(torch.int32), out[perm].view(torch.int32))
    idx = torch.tensor([0, 255, 256, 4095, 9000, 16383], device="cuda")
    out_n, sel_n, _ = L.moe_layer(g, w, x[idx].contiguous(), st, logits=logits[idx].contiguous(), wide=False)
    assert st.read() == 0 and (sel[idx] == sel_n).all()
    assert rel_l2(out[idx].cpu().numpy(), out_n.cpu().numpy()) <= 5e-4
    hw, _ = wl.host_copy()
    Lp = port.layer(wl.spec, hw, allow_q4k=True)
    some = torch.arange(16, device="cuda") * 1023 + 7                       # 16 rows across the batch: 128 pairs + 16 shared
    rc, want, sel0, _ = port.moe_tokens(Lp, x[some].cpu().numpy(), logits=logits[some].cpu().numpy(), threads=min(16, os.cpu_count() or 8))
    assert rc == 0 and (sel[some].cpu().numpy() == sel0).all()
    got = out[some].cpu().numpy()
    assert rel_l2(got, want) <= 1e-3
    assert (np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)).max() <= 4e-3


@pytest.mark.parametrize("world,tokens,topk,experts", [(8, 300, 8, 256), (2, 64, 6, 64), (4, 1, 4, 16)])
def test_ep_dispatch_matches_the_tensor_formulation(L, world, tokens, topk, experts):
    """yvex_b200_ep_dispatch against the stable-argsort formulation the layer uses without it."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(tokens)
    per_rank, H = experts // world, 256
    sel = torch.stack([torch.randperm(experts, device="cuda", generator=g)[:topk] for _ in range(tokens)]).to(torch.int32)
    wts = torch.rand((tokens, topk), device="cuda", generator=g)
    xh = torch.randn((tokens, H), device="cuda", generator=g).to(torch.float16)
    st = L.Status()
    send_rows, meta, inverse, counts = L.ep_dispatch(xh, sel, wts, per_rank, world, st)
    assert st.read() == 0
    dest = (sel // per_rank).reshape(-1).to(torch.int64)
    order = torch.argsort(dest, stable=True)
    assert torch.equal(counts, torch.bincount(dest, minlength=world))
    assert torch.equal(send_rows, xh.index_select(0, torch.div(order, topk, rounding_mode="floor")))
    want_meta = torch.stack(((sel % per_rank).reshape(-1), wts.reshape(-1).view(torch.int32)), dim=1).index_select(0, order)
    assert torch.equal(meta, want_meta)
    want_inv = torch.empty_like(order)
    want_inv[order] = torch.arange(order.numel(), device="cuda")
    assert torch.equal(inverse.to(torch.int64), want_inv)
    # an expert id outside world * per_rank raises the argument status instead of indexing past the bins
    bad = sel.clone()
    bad[0, 0] = experts
    L.ep_dispatch(xh, bad, wts, per_rank, world, st)
    torch.cuda.synchronize()
    assert st.read() == 2


@pytest.mark.parametrize("rows,experts,hidden", [(1, 4, 256), (7, 9, 260), (9, 8, 1024), (17, 256, 512), (333, 64, 4096), (1201, 72, 256),
                                                 (5, 6, 258)])
def test_router_projection_tiles(L, rows, experts, hidden):
    """8 x 8 tiles with ragged ends, rows split over four warps or not (from 1184 tiles on), and the width that takes the
    dot-by-dot kernel. Sums are doubles in another order than numpy's and rounded once: one f32 step."""
    rng = np.random.default_rng(rows)
    x, router = rng.normal(size=(rows, hidden)).astype(np.float32), rng.normal(0, 0.02, (experts, hidden)).astype(np.float32)
    spec = synth.MoELayerSpec(hidden, experts, min(4, experts), 256)
    st = L.Status()
    sel, w, logits = L.moe_route(L.geometry_of(spec), L.weights_of({"router": dev(router)}), st, rows_f32=dev(x))
    assert st.read() == 0
    want = x.astype(np.float64) @ router.astype(np.float64).T
    assert np.allclose(logits.cpu().numpy(), want, rtol=2.0 ** -23, atol=1e-12)


@pytest.mark.parametrize("gate,down,hidden,inter", [(synth.IQ2_XXS, synth.Q4_K, 512, 256), (synth.IQ2_XXS, synth.Q2_K, 1280, 768),
                                                    (synth.Q4_K, synth.IQ2_XXS, 256, 512), (synth.Q2_K, synth.Q2_K, 768, 1280)])
def test_grouped_gemm_tile_edges(L, gate, down, hidden, inter):
    """Group sizes around every edge of a tile - the 16 columns of an MMA, the 32- and 64-row boxes, one, two and three column
    blocks of equal width - with one to five superblocks along K (rows that start on every 16-byte phase), against 64 bits over
    the decoded weights with the layer's two bf16 roundings: 1e-3, the bound of the layer outputs."""
    import torch
    counts = [0, 1, 15, 16, 17, 31, 33, 64, 65, 97, 128, 129, 192, 193, 224, 225, 256, 257, 448, 449, 700]
    E = len(counts)
    spec = synth.MoELayerSpec(hidden, E, 2, inter, gate_qtype=gate, down_qtype=down)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(hidden)
    from yvex_b200.workloads import device_blocks
    t = {n: device_blocks(torch, q, r, w, gen, "cuda") for n, q, r, w in (
        ("gate", gate, E * inter, hidden), ("up", gate, E * inter, hidden), ("down", down, E * hidden, inter),
        ("shared_gate", gate, inter, hidden), ("shared_up", gate, inter, hidden), ("shared_down", down, hidden, inter))}
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts)] + [torch.full((130,), -1, dtype=torch.int32)])
    ids = ids[torch.randperm(ids.numel(), generator=torch.Generator().manual_seed(1))].cuda()
    P = ids.numel()
    x = torch.randn((P, hidden), device="cuda", generator=gen).to(torch.bfloat16)
    w = torch.rand(P, device="cuda", generator=gen) + 0.5
    st = L.Status()
    y = L.moe_expert_rows(L.geometry_of(spec), L.weights_of(t), x.half(), ids, w, st)
    assert st.read() == 0
    want = torch.empty((P, hidden), dtype=torch.float64, device="cuda")
    for e in list(range(E)) + [-1]:
        rows = (ids == e).nonzero()[:, 0]
        if not rows.numel():
            continue
        part = lambda n, q, r, c: L.dequant_rows(q, (t["shared_" + n] if e < 0 else t[n].reshape(E, -1)[e]).contiguous(), r, c, st).double()  # noqa: E731
        g, u = x[rows].double() @ part("gate", gate, inter, hidden).T, x[rows].double() @ part("up", gate, inter, hidden).T
        g, u = g.clamp(max=spec.limit), u.clamp(-spec.limit, spec.limit)
        mid = (g * torch.sigmoid(g) * u * w[rows].double()[:, None]).to(torch.bfloat16).double()
        want[rows] = (mid @ part("down", down, hidden, inter).T).to(torch.bfloat16).double()
    for e in list(range(E)) + [-1]:
        rows = (ids == e).nonzero()[:, 0]
        if rows.numel():
            assert rel_l2(y[rows].float().cpu().numpy(), want[rows].cpu().numpy()) <= 1e-3, (e, rows.numel())


@pytest.mark.parametrize("hidden,inter", [(6400, 512), (8192, 256)])
def test_decode_layer_with_long_q8_0_rows(L, hidden, inter):
    """Q8_0 rows of more than about 6 K weights go through the decode layer's gate and up launch in groups of eight (rows of down
    are at most 4096): against 64 bits over the decoded weights with the layer's bf16 roundings."""
    import torch
    from yvex_b200.workloads import device_blocks
    E, k, T = 3, 2, 5
    spec = synth.MoELayerSpec(hidden, E, k, inter, gate_qtype=synth.Q8_0, down_qtype=synth.Q8_0)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(hidden)
    shapes = dict(gate=(inter, hidden), up=(inter, hidden), down=(hidden, inter))
    t = {n: device_blocks(torch, synth.Q8_0, E * r, w, gen, "cuda") for n, (r, w) in shapes.items()}
    t.update({"shared_" + n: device_blocks(torch, synth.Q8_0, r, w, gen, "cuda") for n, (r, w) in shapes.items()})
    x, logits, st = torch.randn((T, hidden), device="cuda", generator=gen), torch.randn((T, E), device="cuda", generator=gen), L.Status()
    out, sel, wts = L.moe_layer(L.geometry_of(spec), L.weights_of(t), x, st, logits=logits)
    assert st.read() == 0
    rows = x.to(torch.bfloat16).double()

    def expert(e, row, weight):
        part = lambda n: L.dequant_rows(synth.Q8_0, (t["shared_" + n] if e < 0 else t[n].reshape(E, -1)[e]).contiguous(), *shapes[n], st).double()  # noqa: E731
        g, u = part("gate") @ row, part("up") @ row
        g, u = g.clamp(max=spec.limit), u.clamp(-spec.limit, spec.limit)
        mid = (g * torch.sigmoid(g) * u * weight).to(torch.bfloat16).double()
        return (part("down") @ mid).to(torch.bfloat16).float()

    for r in range(T):
        routed = torch.zeros(hidden, device="cuda")
        for p in range(k):
            routed += expert(int(sel[r, p]), rows[r], float(wts[r, p]))
        want = (routed + expert(-1, rows[r], 1.0)).to(torch.bfloat16).float()
        assert rel_l2(out[r].cpu().numpy(), want.cpu().numpy()) <= 1e-3


def test_calls_launched_programmatically_replay_from_a_graph(L):
    """The wide layer, attention and a matvec of several rows captured together: a replay on other inputs in the same buffers gives
    what the calls give, bit for bit (captured programmatic launches keep their order)."""
    import torch
    from yvex_b200.workloads import device_blocks
    H, I, E, k, T = 512, 256, 8, 2, 300
    spec = synth.MoELayerSpec(H, E, k, I, down_qtype=synth.Q2_K)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    q = {n: spec.gate_qtype if n != "down" else spec.down_qtype for n in ("gate", "up", "down")}
    shapes = dict(gate=(I, H), up=(I, H), down=(H, I))
    t = {n: device_blocks(torch, q[n], E * r, w, gen, "cuda") for n, (r, w) in shapes.items()}
    t.update({"shared_" + n: device_blocks(torch, q[n], r, w, gen, "cuda") for n, (r, w) in shapes.items()})
    t["router"] = 0.02 * torch.randn((E, H), device="cuda", generator=gen)
    geometry, weights, st = L.geometry_of(spec), L.weights_of(t), L.Status()
    x, out = torch.empty((T, H), device="cuda"), torch.empty((T, H), device="cuda")
    sel, wts = torch.empty((T, k), dtype=torch.int32, device="cuda"), torch.empty((T, k), device="cuda")
    ws = torch.empty(L.moe_workspace_bytes(geometry, T, True), dtype=torch.uint8, device="cuda")
    qa, key, val = (torch.empty(s, dtype=torch.bfloat16, device="cuda") for s in ((2, 8, 128), (2, 2, 700, 128), (2, 2, 700, 128)))
    aws = torch.empty(int(L.lib.yvex_b200_attention_workspace_bytes(2, 8, 2, 128, 700)), dtype=torch.uint8, device="cuda")
    att = torch.empty((2, 8, 128), device="cuda")
    head = device_blocks(torch, synth.Q4_K, 32768, H, gen, "cuda")
    y = torch.empty((8, 32768), device="cuda")

    def fill():
        x.normal_(generator=gen)
        for v in (qa, key, val):
            v.normal_(generator=gen)

    def calls():
        L.moe_layer(geometry, weights, x, st, wide=True, workspace=ws, out=out, selected=sel, wts=wts)
        L.attention_gqa_decode(qa, key, val, 650, 128 ** -0.5, st, workspace=aws, out=att)
        L.gemv(synth.Q4_K, head, 32768, H, out[:8], st, out=y)
        return [v.clone() for v in (out, sel, wts, att, y)]

    fill()
    calls()                                             # attributes of the kernels are set by their first launch
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        calls()
    for _ in range(2):
        fill()
        want = calls()
        for v in (out, sel, wts, att, y):
            v.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert st.read() == 0
        assert all(torch.equal(a, b) for a, b in zip(want, (out, sel, wts, att, y)))
