"""GPU parity tests: every kernel is driven through the C-ABI of libyvex_b200.so and compared with
the CPU oracle on the same seeded inputs (bit-exact for dequantization and expert selection,
stated tolerances for floating-point results), plus the frozen outputs of the unmodified reference
in tests/golden/. Tolerances:
  * matvec: |gpu - cpu| <= 1e-5 * (1 + |cpu|) scaled by the row's sum |w*x| bound, the
    reference's own CUDA-vs-CPU matvec bound (tests/unit/cuda/quant_qtype.c:262-264);
  * MoE layer outputs: relative L2 <= 1e-3 against the CPU path, identical expert selection
    (tests/live/moe_deepseek.c:223-241);
  * attention: relative L2 <= 1e-4.
"""
import numpy as np
import pytest

from golden_cases import CASES, attention_inputs, layer_inputs
from golden.make_golden import iq2_exhaustive_blocks
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


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def matvec_close(got, want, w_dec, x):
    """1e-5 * (1 + |ref|) plus the f32 accumulation allowance on sum |w*x|."""
    bound = 1e-5 * (1.0 + np.abs(want)) + 2e-6 * (np.abs(w_dec.astype(np.float64)) @ np.abs(x.astype(np.float64)))
    return np.abs(got.astype(np.float64) - want.astype(np.float64)) <= bound


# ---- dequantization: bit exact -------------------------------------------------------------

@pytest.mark.parametrize("name", list(CASES["matvec"]))
def test_dequant_bit_exact_vs_frozen_reference(L, golden, name):
    qtype, rows, width, seed = CASES["matvec"][name]
    w = synth.random_blocks(qtype, rows, width, seed)
    st = L.Status()
    out = L.dequant_rows(qtype, dev(w), rows, width, st).cpu().numpy()
    assert st.read() == 0
    assert (bits(out) == golden[f"decode_{name}"]).all()


def test_dequant_iq2_xxs_all_codes_bit_exact(L, golden):
    blocks = iq2_exhaustive_blocks()
    st = L.Status()
    out = L.dequant_rows(synth.IQ2_XXS, dev(blocks), blocks.shape[0], 256, st).cpu().numpy()
    assert st.read() == 0
    assert (bits(out) == golden["decode_iq2_exhaustive"]).all()


def test_dequant_q4_k_matches_restatement(L, port):
    w = synth.random_blocks(synth.Q4_K, 9, 1024, 5)
    rc, want = port.decode_rows(synth.Q4_K, w, 9, 1024, allow_q4k=True)
    st = L.Status()
    out = L.dequant_rows(synth.Q4_K, dev(w), 9, 1024, st).cpu().numpy()
    assert rc == 0 and st.read() == 0 and (bits(out) == bits(want)).all()


def test_mxfp4_decode_and_matvec(L, port):
    """MXFP4 (the other block qtype the reference decodes): the golden block of tests/unit/quant_numeric.c:529-540,
    random blocks bit-exact against the pinned port, the E8M0 NaN code refused, and the matvec."""
    blk = np.zeros((1, 17), np.uint8)
    blk[0, 0], blk[0, 1:] = 127, 0x21
    st = L.Status()
    out = L.dequant_rows(synth.MXFP4, dev(blk), 1, 32, st).cpu().numpy()[0]
    assert st.read() == 0 and (out[:16] == 0.5).all() and (out[16:] == 1.0).all()
    rows, width = 37, 1024
    w = synth.random_blocks(synth.MXFP4, rows, width, 9)
    rc, want = port.decode_rows(synth.MXFP4, w, rows, width)
    got = L.dequant_rows(synth.MXFP4, dev(w), rows, width, st).cpu().numpy()
    assert rc == 0 and st.read() == 0 and (bits(got) == bits(want)).all()
    x = np.random.default_rng(10).standard_normal(width).astype(np.float32)
    rc, y0 = port.matvec(synth.MXFP4, w, rows, width, x, threads=4)
    y = L.gemv(synth.MXFP4, dev(w), rows, width, dev(x), st).cpu().numpy()[0]
    assert rc == 0 and st.read() == 0 and matvec_close(y, y0, want, x).all()
    bad = w.copy()
    bad[3, 17] = 0xFF
    L.dequant_rows(synth.MXFP4, dev(bad), rows, width, st)
    assert st.read() == 1
    st.reset()
    L.gemv(synth.MXFP4, dev(bad), rows, width, dev(x), st)
    assert st.read() == 1
    # scale code 0 (2^-128, a subnormal) and negative zeros (code 8) in the streaming matvec
    edge = w.copy()
    edge[:, 0] = 0
    edge[5, 1:17] = 0x88
    edge[6, 17 * 3] = 200
    _, dec = port.decode_rows(synth.MXFP4, edge, rows, width)
    rc, y0 = port.matvec(synth.MXFP4, edge, rows, width, x, threads=4)
    st.reset()
    y = L.gemv(synth.MXFP4, dev(edge), rows, width, dev(x), st).cpu().numpy()[0]
    assert rc == 0 and st.read() == 0 and matvec_close(y, y0, dec, x).all()


def test_malformed_scale_sets_status_word(L):
    w = synth.random_blocks(synth.IQ2_XXS, 2, 256, 3)
    w[1, 0:2] = [0x00, 0xBC]          # d = -1.0: the reference refuses negative scales
    st = L.Status()
    L.dequant_rows(synth.IQ2_XXS, dev(w), 2, 256, st)
    assert st.read() == 1


# ---- matvec ----------------------------------------------------------------------------------

@pytest.mark.parametrize("name", list(CASES["matvec"]))
def test_gemv_vs_frozen_reference(L, golden, port, name):
    qtype, rows, width, seed = CASES["matvec"][name]
    w = synth.random_blocks(qtype, rows, width, seed)
    x = np.random.default_rng(seed + 1).standard_normal(width).astype(np.float32)
    st = L.Status()
    y = L.gemv(qtype, dev(w), rows, width, dev(x), st).cpu().numpy()[0]
    want = golden[f"matvec_{name}"].view(np.float32)
    dec = golden[f"decode_{name}"].view(np.float32)
    assert st.read() == 0
    assert matvec_close(y, want, dec, x).all(), np.abs(y - want).max()


@pytest.mark.parametrize("qtype,rows,width", [(synth.IQ2_XXS, 4096, 4096), (synth.IQ2_XXS, 1, 256),
                                              (synth.IQ2_XXS, 13, 7168), (synth.IQ2_XXS, 100, 1536),
                                              (synth.Q4_K, 257, 1536), (synth.Q4_K, 64, 2048),
                                              (synth.Q8_0, 300, 4096), (synth.Q2_K, 129, 2048), (synth.Q2_K, 4096, 4096),
                                              (synth.Q2_K, 13, 7168), (synth.Q2_K, 100, 1536), (synth.Q2_K, 1, 256),
                                              (synth.Q8_0, 4096, 4096), (synth.Q8_0, 37, 1280), (synth.Q8_0, 5, 256),
                                              (synth.Q8_0, 3000, 7168)])
def test_gemv_vs_oracle_shapes(L, port, qtype, rows, width):
    """Config-1 shape (4096x4096 IQ2_XXS, f32 N(0,1) activation) and ragged row counts / widths
    that exercise tile tails and rows that start on 8-byte boundaries only."""
    w = synth.random_blocks(qtype, rows, width, 1000 + rows)
    x = np.random.default_rng(rows).standard_normal(width).astype(np.float32)
    rc, want = port.matvec(qtype, w, rows, width, x, threads=8, allow_q4k=True)
    _, dec = port.decode_rows(qtype, w, rows, width, allow_q4k=True)
    st = L.Status()
    y = L.gemv(qtype, dev(w), rows, width, dev(x), st).cpu().numpy()[0]
    assert rc == 0 and st.read() == 0
    ok = matvec_close(y, want, dec, x)
    assert ok.all(), (np.abs(y - want).max(), int((~ok).sum()))


@pytest.mark.parametrize("qtype,rows,width", [(synth.F32, 64, 4096), (synth.F16, 300, 1536), (synth.BF16, 37, 7168),
                                              (synth.F32, 5, 96), (synth.F16, 1, 8), (synth.BF16, 129, 250)])
def test_gemv_scalar_qtypes_vs_oracle(L, port, qtype, rows, width):
    """F32 / F16 / BF16 rows (router weights and coefficient tensors are stored this way) on the
    warp-per-row kernel, widths that are no multiple of 32 included."""
    rng = np.random.default_rng(rows * 31 + width)
    wf = (rng.standard_normal((rows, width)) * 0.02).astype(np.float32)
    if qtype == synth.F32:
        enc = wf.view(np.uint8)
    elif qtype == synth.F16:
        enc = wf.astype(np.float16).view(np.uint8)
    else:
        enc = synth.bf16_bits(wf).reshape(rows, width).view(np.uint8)
    enc = np.ascontiguousarray(enc).reshape(rows, -1)
    x = rng.standard_normal(width).astype(np.float32)
    rc, want = port.matvec(qtype, enc, rows, width, x, threads=4)
    rcd, dec = port.decode_rows(qtype, enc, rows, width)
    st = L.Status()
    out = L.dequant_rows(qtype, dev(enc), rows, width, st).cpu().numpy()
    y = L.gemv(qtype, dev(enc), rows, width, dev(x), st).cpu().numpy()[0]
    assert rc == 0 and rcd == 0 and st.read() == 0
    assert (bits(out) == bits(dec)).all()
    assert matvec_close(y, want, dec, x).all(), np.abs(y - want).max()


@pytest.mark.parametrize("qtype", [synth.IQ2_XXS, synth.Q8_0])
def test_gemv_input_rows_additive_and_bf16(L, port, qtype):
    rows, width = 40, 1024
    w = synth.random_blocks(qtype, rows, width, 77)
    rng = np.random.default_rng(78)
    x = rng.standard_normal((3, width)).astype(np.float32)
    add = rng.standard_normal((3, rows)).astype(np.float32)
    st = L.Status()
    y = L.gemv(qtype, dev(w), rows, width, dev(x), st, additive=dev(add), round_bf16=True).cpu().numpy()
    assert st.read() == 0
    for i in range(3):
        _, want = port.matvec(qtype, w, rows, width, x[i])
        want = synth.bf16_round(want + add[i])
        assert rel_l2(y[i], want) < 4e-3 and (np.abs(y[i] - want) <= 2 ** -7 * np.abs(want) + 1e-6).all()
        assert (synth.bf16_round(y[i]).view(np.uint32) == y[i].view(np.uint32)).all()


@pytest.mark.parametrize("qtype,count,rows,width", [(synth.IQ2_XXS, 5, 300, 4096), (synth.Q4_K, 3, 77, 1536), (synth.Q8_0, 4, 33, 2048),
                                                    (synth.IQ2_XXS, 40, 16, 256), (synth.Q2_K, 3, 20, 512), (synth.Q2_K, 6, 300, 2048),
                                                    (synth.MXFP4, 2, 20, 512), (synth.MXFP4, 3, 77, 1536), (synth.MXFP4, 2, 300, 4096),
                                                    (synth.MXFP4, 1, 40, 8192), (synth.MXFP4, 2, 20, 768)])
def test_gemv_batch_vs_oracle(L, port, qtype, count, rows, width):
    """Independent matrices with their own input rows in one launch (ragged tiles, tiles of different
    matrices inside one CTA's task range, a qtype that falls back to one matvec per matrix)."""
    w = synth.random_blocks(qtype, rows * count, width, 500 + rows)
    rng = np.random.default_rng(count)
    x = (rng.standard_normal((count, width)) * np.logspace(-3, 2, count)[:, None]).astype(np.float32)      # rows of very different scale
    add = rng.standard_normal((count, rows)).astype(np.float32)
    st = L.Status()
    y = L.gemv_batch(qtype, dev(w.reshape(-1)), count, rows, width, dev(x), st).cpu().numpy()
    ya = L.gemv_batch(qtype, dev(w.reshape(-1)), count, rows, width, dev(x), st, additive=dev(add)).cpu().numpy()
    assert st.read() == 0
    for m in range(count):
        wm = w[m * rows:(m + 1) * rows]
        rc, want = port.matvec(qtype, wm, rows, width, x[m], threads=4, allow_q4k=True)
        _, dec = port.decode_rows(qtype, wm, rows, width, allow_q4k=True)
        assert rc == 0 and matvec_close(y[m], want, dec, x[m]).all(), (m, np.abs(y[m] - want).max())
        assert matvec_close(ya[m] - add[m], want, dec, x[m]).all() or np.abs(ya[m] - (want + add[m])).max() <= 1e-5 * (1 + np.abs(want + add[m]).max())


def test_gemv_streaming_kernel_edge_cases(L, port):
    """A zero input row, one huge element among tiny ones (the fixed-point planes follow the row's largest
    magnitude), a malformed block scale in an existing row, and a non-finite input."""
    rows, width = 50, 1024
    w = synth.random_blocks(synth.IQ2_XXS, rows, width, 61)
    st = L.Status()
    y = L.gemv(synth.IQ2_XXS, dev(w), rows, width, dev(np.zeros(width, np.float32)), st).cpu().numpy()[0]
    assert st.read() == 0 and not y.any()
    x = (np.random.default_rng(2).standard_normal(width) * 1e-3).astype(np.float32)
    x[17] = 900.0
    y = L.gemv(synth.IQ2_XXS, dev(w), rows, width, dev(x), st).cpu().numpy()[0]
    rc, want = port.matvec(synth.IQ2_XXS, w, rows, width, x)
    _, dec = port.decode_rows(synth.IQ2_XXS, w, rows, width)
    assert rc == 0 and st.read() == 0 and matvec_close(y, want, dec, x).all()
    bad = w.copy()
    bad[49, 66:68] = [0x00, 0xFC]                    # d = -inf in the second block of the last row
    L.gemv(synth.IQ2_XXS, dev(bad), rows, width, dev(x), st)
    assert st.read() == 1
    st.reset()
    x[5] = np.nan
    L.gemv(synth.IQ2_XXS, dev(w), rows, width, dev(x), st)
    assert st.read() == 1


def test_gemv_linearity_at_full_size(L):
    """Size-independent property: W(a*x1 + x2) == a*W(x1) + W(x2) up to f32 rounding."""
    rows = width = 4096
    w = dev(synth.random_blocks(synth.IQ2_XXS, rows, width, 4242))
    rng = np.random.default_rng(1)
    x1, x2 = rng.standard_normal(width).astype(np.float32), rng.standard_normal(width).astype(np.float32)
    st = L.Status()
    y1 = L.gemv(synth.IQ2_XXS, w, rows, width, dev(x1), st).cpu().numpy()[0]
    y2 = L.gemv(synth.IQ2_XXS, w, rows, width, dev(x2), st).cpu().numpy()[0]
    y3 = L.gemv(synth.IQ2_XXS, w, rows, width, dev((2.0 * x1 + x2).astype(np.float32)), st).cpu().numpy()[0]
    assert st.read() == 0 and rel_l2(y3, 2.0 * y1 + y2) < 1e-5


def test_gemv_refuses_unsupported_qtype_without_touching_status(L):
    import torch
    st = L.Status()
    enc = torch.zeros(110 * 8, dtype=torch.uint8, device="cuda")
    with pytest.raises(L.YvexError) as e:
        L.gemv(11, enc, 8, 256, torch.zeros(256, device="cuda"), st)
    assert e.value.code == -5 and st.read() == 0


# ---- router ----------------------------------------------------------------------------------

def test_router_known_answers_on_device(L):
    # tests/unit/runtime_moe.c:111-171
    spec = synth.MoELayerSpec(4, 4, 2, 2)
    router = np.array([[1, 0, 0, 0], [2, 0, 0, 0], [2, 0, 0, 0], [0, 0, 0, 0]], np.float32)
    x = np.array([[1, 0, 0, 0]], np.float32)
    st = L.Status()
    g = L.geometry_of(spec)
    sel, w, _ = L.moe_route(g, L.weights_of({"router": dev(router), "bias": dev(np.array([5, 0, 0, 0], np.float32))}),
                            st, rows_f32=dev(x))
    a, b = np.sqrt(np.log1p(np.exp(1.0))), np.sqrt(2 + np.log1p(np.exp(-2.0)))
    assert sel.cpu().numpy().tolist() == [[0, 1]]
    assert np.allclose(w.cpu().numpy(), [[a / (a + b) * 1.5, b / (a + b) * 1.5]], atol=1e-6)
    sel, _, _ = L.moe_route(g, L.weights_of({"router": dev(router)}), st, rows_f32=dev(x))
    assert sel.cpu().numpy().tolist() == [[1, 2]] and st.read() == 0
    table = dev(np.array([3, 1], np.int32))
    gh = L.geometry_of(spec, router_class=0, hash_rows=8, hash_stored_rows=1)
    sel, _, _ = L.moe_route(gh, L.weights_of({"router": dev(router), "hash_table": table}), st, rows_f32=dev(x),
                            token_ids=dev(np.array([4], np.uint32)))
    assert sel.cpu().numpy().tolist() == [[3, 1]] and st.read() == 0
    L.moe_route(gh, L.weights_of({"router": dev(router), "hash_table": dev(np.array([3, 3], np.int32))}), st,
                rows_f32=dev(x), token_ids=dev(np.array([4], np.uint32)))
    assert st.read() == 2            # duplicate selection refuses
    st.reset()
    L.moe_route(gh, L.weights_of({"router": dev(router), "hash_table": table}), st, rows_f32=dev(x),
                token_ids=dev(np.array([8], np.uint32)))
    assert st.read() == 2            # out-of-vocabulary token refuses


@pytest.mark.parametrize("experts,topk,rows", [(64, 6, 257), (256, 8, 512), (7, 3, 5)])
def test_router_selection_identical_to_oracle(L, port, experts, topk, rows):
    spec = synth.MoELayerSpec(256, experts, topk, 256)
    rng = np.random.default_rng(experts)
    logits = rng.standard_normal((rows, experts)).astype(np.float32)
    logits[0, :] = 0.25                        # full tie: lowest indices must win
    bias = (rng.standard_normal(experts) * 0.1).astype(np.float32)
    bias[:topk + 1] = 0.5                      # ... among the experts the bias leaves tied
    st = L.Status()
    sel, w, _ = L.moe_route(L.geometry_of(spec), L.weights_of({"bias": dev(bias)}), st, logits=dev(logits))
    sel, w = sel.cpu().numpy(), w.cpu().numpy()
    Lp = port.layer(spec, {}, bias=bias)
    for r in range(rows):
        rc, s0, w0, _, _ = port.route(Lp, logits[r])
        assert rc == 0 and sel[r].tolist() == s0.tolist()
        assert np.abs(w[r] - w0).max() <= 2e-7
    assert st.read() == 0 and sel[0].tolist() == list(range(topk))


# ---- expert worklist ---------------------------------------------------------------------------

@pytest.mark.parametrize("rows,topk,experts", [(1, 6, 64), (62, 8, 256), (5, 3, 7), (300, 8, 256), (2048, 6, 64), (16384, 8, 256)])
def test_expert_worklist_matches_the_reference_order(L, port, rows, topk, experts):
    """The device sort against the reference builder's order (src/graph/worklist.c:369-441): buckets
    ascending by expert, populated experts only, pairs ascending within a bucket, source row = pair /
    topk, destination row = pair; and the summary the reference's device builder publishes
    (src/backend/cuda/moe_kernels.cu:294-397). Narrow batches run the one-CTA kernel, wide ones the
    count / plan / scatter kernels of the grouped-GEMM path itself."""
    import torch
    rng = np.random.default_rng(rows + experts)
    sel = np.stack([rng.permutation(experts)[:topk] for _ in range(rows)]).astype(np.int32)
    if rows > 4:
        sel[sel == 3] = 4 if topk < experts - 1 else 3            # leave expert 3 (nearly) empty
        sel = np.where((sel == 4) & (np.cumsum(sel == 4, axis=1) > 1), 3, sel).astype(np.int32)
    st = L.Status()
    tc_min, width = 4, 16
    got = L.expert_worklist(torch.from_numpy(sel).cuda(), experts, st, tensor_core_minimum=tc_min, admitted_width=width,
                            provenance=3 if rows > 62 else 2)
    rc, order, src, be, bo, bc = port.worklist(sel.astype(np.uint64), experts)
    assert rc == 0 and st.read() == 0
    assert (got["order"] == order).all() and (got["source_rows"] == src).all() and (got["destination_rows"] == order).all()
    assert (got["expert_ids"] == be).all() and (got["bucket_offsets"] == bo).all() and (got["bucket_populations"] == bc).all()
    o = got["observation"]
    pairs = rows * topk
    assert (o.schema_version, o.worklist_count, o.pair_count, o.bucket_count) == (1, 1, pairs, len(be))
    assert o.maximum_bucket_population == bc.max()
    eligible = int(bc[bc >= tc_min].sum())
    assert o.tensor_core_eligible_pairs == eligible and o.narrow_pairs == pairs - eligible and o.tensor_core_executed_pairs == 0
    assert o.tail_rows == int(sum((width - n % width) % width for n in bc[bc >= tc_min]))
    assert list(o.population_histogram) == np.bincount(np.minimum(bc, 16), minlength=17).tolist()
    assert list(o.width_histogram) == [1 if i == min(rows, 16) else 0 for i in range(17)]
    assert list(o.provenance_counts) == [1 if i == (3 if rows > 62 else 2) else 0 for i in range(5)]


def test_expert_worklist_refuses_foreign_expert_ids(L):
    import torch
    st = L.Status()
    sel = torch.tensor([[0, 1], [2, 9]], dtype=torch.int32, device="cuda")
    L.expert_worklist(sel, 8, st)
    assert st.read() == 2
    st.reset()
    big = torch.randint(0, 8, (4096, 2), dtype=torch.int32, device="cuda")
    big[77, 1] = 8
    L.expert_worklist(big, 8, st)
    assert st.read() == 2


# ---- MoE layer -------------------------------------------------------------------------------

def run_layer(L, spec, weights, router, x, logits, wide=False):
    t = {k: dev(v.reshape(-1)) for k, v in weights.items()}
    if router is not None:
        t["router"] = dev(router)
    st = L.Status()
    out, sel, w = L.moe_layer(L.geometry_of(spec), L.weights_of(t), dev(x), st,
                              logits=None if logits is None else dev(logits), wide=wide)
    return out.cpu().numpy(), sel.cpu().numpy(), w.cpu().numpy(), st.read()


@pytest.mark.parametrize("name", list(CASES["layer"]))
def test_moe_decode_layer_vs_frozen_reference(L, golden, name):
    spec, weights, router, x, logits = layer_inputs(name)
    out, sel, w, status = run_layer(L, spec, weights, router, x, logits)
    assert status == 0
    assert (sel == golden[f"layer_{name}_sel"]).all()
    assert np.abs(w - golden[f"layer_{name}_w"].view(np.float32)).max() <= 2e-7
    want = golden[f"layer_{name}_out"].view(np.float32)
    assert rel_l2(out, want) <= 1e-3, rel_l2(out, want)


@pytest.mark.parametrize("name", ["small_router", "c2_shape"])
def test_moe_decode_layer_q4_k_down_vs_restatement(L, port, name):
    """Config 2 as specified (IQ2_XXS gate/up, Q4_K down). Q4_K has no reference decoder: the
    check is against this repository's restatement (reference-unpinned)."""
    spec, weights, router, x, logits = layer_inputs(name, down_qtype=synth.Q4_K)
    Lp = port.layer(spec, weights, router=router, allow_q4k=True)
    rc, want, sel0, w0 = port.moe_tokens(Lp, x, logits=logits, threads=8)
    out, sel, w, status = run_layer(L, spec, weights, router, x, logits)
    assert rc == 0 and status == 0 and (sel == sel0).all()
    assert rel_l2(out, want) <= 1e-3, rel_l2(out, want)


def test_moe_layer_outputs_are_bf16_values_and_rows_independent(L):
    spec, weights, router, x, logits = layer_inputs("small_logits")
    out, sel, _, status = run_layer(L, spec, weights, router, x, logits)
    assert status == 0 and (synth.bf16_round(out).view(np.uint32) == out.view(np.uint32)).all()
    out1, sel1, _, _ = run_layer(L, spec, weights, router, x[2:3], logits[2:3])
    assert (out1.view(np.uint32) == out[2:3].view(np.uint32)).all() and (sel1 == sel[2:3]).all()


def test_moe_nonfinite_input_sets_status(L):
    spec, weights, router, x, logits = layer_inputs("small_logits")
    x = x.copy()
    x[1, 7] = np.inf
    assert run_layer(L, spec, weights, router, x, logits)[3] == 1


# ---- attention -------------------------------------------------------------------------------

@pytest.mark.parametrize("name", list(CASES["attention"]))
def test_gqa_decode_vs_frozen_reference(L, golden, name):
    import torch
    q, k, v, pos, scale = attention_inputs(name)
    st = L.Status()
    out = L.attention_gqa_decode(dev(q).to(torch.bfloat16), dev(k).to(torch.bfloat16), dev(v).to(torch.bfloat16),
                                 pos, scale, st).cpu().numpy()
    want = golden[f"attention_{name}"].view(np.float32)
    assert st.read() == 0 and rel_l2(out, want) <= 1e-4, rel_l2(out, want)


def test_gqa_decode_long_context_vs_oracle(L, port):
    """Config-4 geometry (32 q / 8 kv heads, d 128) on 2 sessions x 8192 context, plus the
    softmax invariance property at that size: shifting every key by a constant vector along q
    changes all scores by the same amount and must not change the output."""
    import torch
    S, Hq, Hkv, D, ctx = 2, 32, 8, 128, 8192
    rng = np.random.default_rng(99)
    q = synth.bf16_round(rng.standard_normal((S, Hq, D)).astype(np.float32))
    k = synth.bf16_round(rng.standard_normal((S, Hkv, ctx, D)).astype(np.float32))
    v = synth.bf16_round(rng.standard_normal((S, Hkv, ctx, D)).astype(np.float32))
    st = L.Status()
    out = L.attention_gqa_decode(dev(q).to(torch.bfloat16), dev(k).to(torch.bfloat16), dev(v).to(torch.bfloat16),
                                 ctx - 1, D ** -0.5, st).cpu().numpy()
    rc, want = port.attention_gqa_decode(synth.bf16_bits(q).reshape(q.shape), synth.bf16_bits(k).reshape(k.shape),
                                         synth.bf16_bits(v).reshape(v.shape), ctx - 1, D ** -0.5, threads=8)
    assert rc == 0 and st.read() == 0 and rel_l2(out, want) <= 1e-4, rel_l2(out, want)
    half = L.attention_gqa_decode(dev(q).to(torch.bfloat16), dev(k).to(torch.bfloat16), dev(v).to(torch.bfloat16),
                                  ctx // 2, D ** -0.5, st).cpu().numpy()
    rc, want_half = port.attention_gqa_decode(synth.bf16_bits(q).reshape(q.shape), synth.bf16_bits(k).reshape(k.shape),
                                              synth.bf16_bits(v).reshape(v.shape), ctx // 2, D ** -0.5, threads=8)
    assert rel_l2(half, want_half) <= 1e-4


def test_attention_f32_single_head_vs_oracle(L, port):
    rng = np.random.default_rng(8)
    q = rng.standard_normal(64).astype(np.float32)
    k = rng.standard_normal((200, 64)).astype(np.float32)
    v = rng.standard_normal((200, 64)).astype(np.float32)
    st = L.Status()
    for pos, causal in ((199, 1), (57, 1), (57, 0)):
        out, scores, probs = L.attention_f32(dev(q), dev(k), dev(v), pos, 0.125, causal, st)
        rc, want = port.attention_head(q, k, v, pos, 0.125, causal)
        assert rc == 0 and rel_l2(out.cpu().numpy(), want) <= 1e-5
        if causal:
            assert not scores.cpu().numpy()[pos + 1:].any() and not probs.cpu().numpy()[pos + 1:].any()
        assert abs(float(probs.sum()) - 1.0) < 1e-5
    assert st.read() == 0


@pytest.mark.parametrize("heads,n,D", [(4, 37, 64), (8, 300, 512), (2, 0, 128), (3, 9, 1024), (5, 1000, 192)])
def test_sink_attention_reducer_vs_restatement(L, heads, n, D):
    """yvex_b200_attention_sink against the numpy restatement of reduce_head (src/graph/core.c:428-465): f32 results
    agree to 2e-6 relative of the largest row value (the kernel merges per-warp running sums instead of walking the
    rows in order), the bf16-rounded ones differ by at most one bf16 step on a few elements."""
    from oracle_lib import sink_attention
    rng = np.random.default_rng(heads * 1000 + n)
    q = rng.standard_normal((heads, D)).astype(np.float32)
    rows = rng.standard_normal((n, D)).astype(np.float32)
    sinks = rng.standard_normal(heads).astype(np.float32) * 3
    scale = 1.0 / np.sqrt(D)
    st = L.Status()
    got = L.attention_sink(dev(q), dev(rows), dev(sinks), scale, st, round_bf16=False).cpu().numpy()
    want = sink_attention(q, rows, sinks, scale, round_bf16=False)
    assert st.read() == 0 and np.abs(got - want).max() <= 2e-6 * max(1.0, np.abs(rows).max() if n else 1.0)
    got16 = L.attention_sink(dev(q), dev(rows), dev(sinks), scale, st, round_bf16=True).cpu().numpy()
    want16 = sink_attention(q, rows, sinks, scale, round_bf16=True)
    assert (synth.bf16_round(got16).view(np.uint32) == got16.view(np.uint32)).all()
    differ = got16.view(np.uint32) != want16.view(np.uint32)
    assert differ.mean() <= 0.01 and (np.abs(got16 - want16)[differ] <= np.abs(want16)[differ] * 2.0 ** -7 + 1e-30).all()
    if n:
        bad = q.copy()
        bad[0, 1] = np.inf
        L.attention_sink(dev(bad), dev(rows), dev(sinks), scale, st)
        assert st.read() == 1


@pytest.mark.parametrize("dim,group,sessions,kv,visible,context", [(64, 1, 1, 1, 1, 16), (64, 4, 3, 2, 63, 64), (128, 2, 2, 2, 65, 300),
                                                                   (128, 4, 1, 8, 1500, 4096), (256, 4, 1, 1, 4097, 4100),
                                                                   (256, 1, 2, 3, 129, 129), (128, 1, 40, 16, 700, 701)])
def test_gqa_decode_slices_and_block_edges(L, dim, group, sessions, kv, visible, context):
    """One key, slices shorter than a block, slices that stay empty, every group and width: against the
    same contraction in 64 bits. Probabilities carry 16 bits (hi + lo bf16) and sums are f32: 1e-5. The context is larger
    than what is visible, what lies behind it is NaN, and a workspace made for the context serves the prefix."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(dim + visible)
    q = torch.randn((sessions, kv * group, dim), device="cuda", generator=gen).to(torch.bfloat16)
    k, v = (torch.randn((sessions, kv, context, dim), device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2))
    k[:, :, visible:], v[:, :, visible:] = float("nan"), float("nan")
    ws = torch.empty(int(L.lib.yvex_b200_attention_workspace_bytes(sessions, kv * group, kv, dim, context)), dtype=torch.uint8, device="cuda")
    st = L.Status()
    out = L.attention_gqa_decode(q, k, v, visible - 1, dim ** -0.5, st, workspace=ws)
    assert st.read() == 0
    scores = torch.einsum("skgd,skcd->skgc", q.double().reshape(sessions, kv, group, dim), k[:, :, :visible].double()) * dim ** -0.5
    want = torch.einsum("skgc,skcd->skgd", torch.softmax(scores, -1), v[:, :, :visible].double()).reshape(out.shape)
    assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) <= 1e-5
    need = [int(L.lib.yvex_b200_attention_workspace_bytes(sessions, kv * group, kv, dim, c)) for c in range(1, context + 1)]
    assert all(a <= b for a, b in zip(need, need[1:]))


@pytest.mark.parametrize("qtype", [synth.F32, synth.F16, synth.BF16])
@pytest.mark.parametrize("rows,width,inputs", [(2048, 256, 2), (2051, 1000, 3), (2050, 512, 8), (9473, 264, 9), (2049, 8192, 17), (2048, 16, 4),
                                               (4099, 1000, 2), (8195, 264, 4), (14211, 2056, 8), (14209, 4096, 5), (2047, 512, 9)])
def test_gemv_scalar_qtypes_several_inputs(L, qtype, rows, width, inputs):
    """Four matrix rows per warp and two, four or eight inputs per pass: ragged rows, widths below a warp's chunk and a width
    whose eight rows do not fit beside each other, against 64 bits (f32 sums of `width` products: 1e-6), with an additive row
    and with bf16 results (the f32 result rounded)."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows + inputs)
    w = torch.randn((rows, width), device="cuda", generator=gen).to({synth.F32: torch.float32, synth.F16: torch.float16, synth.BF16: torch.bfloat16}[qtype])
    x, st = torch.randn((inputs, width), device="cuda", generator=gen), L.Status()
    y = L.gemv(qtype, w.view(torch.uint8).reshape(-1), rows, width, x, st)
    assert st.read() == 0
    assert rel_l2(y.cpu().numpy(), (x.double() @ w.double().T).cpu().numpy()) <= 1e-6
    add = torch.randn((inputs, rows), device="cuda", generator=gen)
    plus = L.gemv(qtype, w.view(torch.uint8).reshape(-1), rows, width, x, st, additive=add)
    assert torch.equal(plus, y + add)
    assert torch.equal(L.gemv(qtype, w.view(torch.uint8).reshape(-1), rows, width, x, st, additive=add, round_bf16=True), plus.to(torch.bfloat16).float())
    assert st.read() == 0
    x[inputs - 1, width - 1] = float("inf")
    L.gemv(qtype, w.view(torch.uint8).reshape(-1), rows, width, x, st)
    assert st.read() == 1


@pytest.mark.parametrize("qtype", [synth.F32, synth.F16, synth.BF16])
@pytest.mark.parametrize("width,inputs", [(1024, 4), (2048, 8), (4096, 2), (4096, 8), (8192, 4)])
def test_gemv_scalar_several_inputs_lose_no_precision(L, qtype, width, inputs):
    """Rows that share a pass are as close to 64 bits as the same rows one call each: f32 sums of the same products in chains
    that are no longer. 2 % is what the sampled error of 16384 and more results varies by."""
    import torch
    rows, st = 16384, L.Status()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(width)
    w = (torch.randn((rows, width), device="cuda", generator=gen) * 0.02).to({synth.F32: torch.float32, synth.F16: torch.float16, synth.BF16: torch.bfloat16}[qtype])
    x, enc = torch.randn((inputs, width), device="cuda", generator=gen), w.view(torch.uint8).reshape(-1)
    y = L.gemv(qtype, enc, rows, width, x, st).double()
    one = torch.stack([L.gemv(qtype, enc, rows, width, x[i], st)[0] for i in range(inputs)]).double()
    want = x.double() @ w.double().T
    assert st.read() == 0
    error, alone = (float((v - want).norm() / want.norm()) for v in (y, one))
    assert error <= 1.02 * alone, (error, alone)


@pytest.mark.parametrize("qtype", [synth.IQ2_XXS, synth.Q4_K, synth.Q8_0, synth.Q2_K, synth.MXFP4])
@pytest.mark.parametrize("rows,width,inputs", [(17, 512, 2), (33, 1536, 3), (300, 4096, 8), (5, 7168, 5), (64, 1024, 4), (40, 256, 6), (16, 8192, 9),
                                               (65539, 512, 8), (32777, 1536, 7), (16411, 4096, 6), (9001, 5120, 9)])
def test_gemv_block_qtypes_several_inputs(L, qtype, rows, width, inputs):
    """Several input rows against one call per row: small matrices and widths whose planes leave no room for four rows (a pass per
    row), large ones in passes of four, full and ragged passes, ragged tiles, rows and planes of every slicing. Exact integer products and the
    same f32 steps: 1e-6 covers another slicing of K. One non-finite value in the last row is refused."""
    import torch
    if qtype == synth.MXFP4 and width % 512:
        pytest.skip("rows of an odd number of 256-weight units")
    w = dev(synth.random_blocks(qtype, rows, width, rows + width))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(inputs)
    x, add, st = torch.randn((inputs, width), device="cuda", generator=gen), torch.randn((inputs, rows), device="cuda", generator=gen), L.Status()
    scale = torch.logspace(-3, 3, inputs, device="cuda")[:, None]        # every row needs its own
    x, add = x * scale, add * scale
    y = L.gemv(qtype, w, rows, width, x, st, additive=add)
    one = torch.stack([L.gemv(qtype, w, rows, width, x[i], st, additive=add[i])[0] for i in range(inputs)])
    assert st.read() == 0
    for i in range(inputs):
        assert rel_l2(y[i].cpu().numpy(), one[i].cpu().numpy()) <= 1e-6
    x[inputs - 1, width - 1] = float("nan")
    L.gemv(qtype, w, rows, width, x, st)
    assert st.read() == 1


@pytest.mark.parametrize("qtype", [synth.IQ2_XXS, synth.Q4_K, synth.Q8_0, synth.Q2_K, synth.MXFP4])
@pytest.mark.parametrize("width", [1024, 4096, 5120])
@pytest.mark.parametrize("mean", [0.0, 1.0, 3.0])
def test_gemv_several_inputs_lose_no_precision(L, qtype, width, mean):
    """Rows that share a decode are as close to 64 bits over the decoded weights as the same rows one call each, inputs with a
    mean included (the minimum terms of Q4_K and Q2_K and MXFP4's offset then cancel large sums). Both are f32 sums of the same
    exact products in another order; 5 % is what the sampled error of that many results varies by, 2e-8 the f32 result itself."""
    import torch
    rows, inputs = 16395, 7
    w = dev(synth.random_blocks(qtype, rows, width, width))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(width)
    x, st = mean + (0.3 if mean else 1.0) * torch.randn((inputs, width), device="cuda", generator=gen), L.Status()
    y = L.gemv(qtype, w, rows, width, x, st).double()
    one = torch.stack([L.gemv(qtype, w, rows, width, x[i], st)[0] for i in range(inputs)]).double()
    want = x.double() @ L.dequant_rows(qtype, w, rows, width, st).double().T
    assert st.read() == 0
    error, alone = (float((v - want).norm() / want.norm()) for v in (y, one))
    assert error <= 1.05 * alone + 2e-8, (error, alone)


@pytest.mark.parametrize("rows,width,inputs", [(2048, 7168, 1), (8, 8192, 1), (13, 6912, 2), (1, 7936, 5), (149 * 8 + 3, 8192, 1)])
def test_gemv_q8_0_long_rows(L, rows, width, inputs):
    """Rows of which sixteen leave no room for a second stage go in groups of eight: ragged tiles, padded and plain pitches,
    several inputs, against 64 bits (the activation is held to 28 bits: 1e-6)."""
    import torch
    raw = synth.random_blocks(synth.Q8_0, rows, width, rows)
    blocks = raw.reshape(rows, -1, 34)
    w = blocks[:, :, :2].copy().view(np.float16).astype(np.float64) * blocks[:, :, 2:].copy().view(np.int8)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(width)
    x, st = torch.randn((inputs, width), device="cuda", generator=gen), L.Status()
    y = L.gemv(synth.Q8_0, dev(raw), rows, width, x, st)
    assert st.read() == 0 and rel_l2(y.cpu().numpy(), x.cpu().numpy().astype(np.float64) @ w.reshape(rows, width).T) <= 1e-6
