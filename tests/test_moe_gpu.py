"""MoE routing, token movement and the expert layer against the CPU oracle.

Byte-producing kernels (plan, gather + quantise, unpermute of exact data) are compared bit
for bit; the layer itself within the bounds the reference uses for its MoE
(test_kernels.py:94-102: max error < 1e-1 and rms < 1e-2 of max|want|), because one bf16 ulp
of GEMM1 can become a whole e2m1 step after the intermediate requantisation."""

import ml_dtypes
import numpy as np
import pytest
import torch

from oracle import moe as M, nvfp4 as O

pytestmark = pytest.mark.gpu


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _weights(E, h, n, seed):
    rng = np.random.default_rng([seed, 0])
    w1 = (rng.standard_normal((E, 2 * n, h)) * 0.05).astype(np.float32)
    w2 = (rng.standard_normal((E, h, n)) * 0.05).astype(np.float32)
    w1_gs, w2_gs = O.global_scale_for(w1), O.global_scale_for(w2)
    w1_q, w1_sf = O.quantize_nvfp4(w1, w1_gs)
    w2_q, w2_sf = O.quantize_nvfp4(w2, w2_gs)
    w1_alpha = rng.uniform(0.5, 1.5, E).astype(np.float32)
    w2_alpha = rng.uniform(0.5, 1.5, E).astype(np.float32)
    return dict(w1_q=w1_q, w1_sf=w1_sf, w1_gs=w1_gs, w1_alpha=w1_alpha,
                w2_q=w2_q, w2_sf=w2_sf, w2_gs=w2_gs, w2_alpha=w2_alpha)


def _dev_weights(w):
    return dict(w1_q=T(O.pack_e2m1(w["w1_q"])), w1_sf=T(O.e4m3_bytes(O.retile(w["w1_sf"]))),
                w1_gs=T(w["w1_gs"]), w1_alpha=T(w["w1_alpha"]),
                w2_q=T(O.pack_e2m1(w["w2_q"])), w2_sf=T(O.e4m3_bytes(O.retile(w["w2_sf"]))),
                w2_gs=T(w["w2_gs"]), w2_alpha=T(w["w2_alpha"]))


def _close(got, want, nonzero_fraction=0.5):
    scale = max(np.abs(want).max(), 1e-6)
    rel = np.abs(got - want).max() / scale
    rms = np.sqrt(np.mean((got - want) ** 2)) / scale
    assert rel < 1e-1 and rms < 1e-2, (rel, rms)
    assert np.count_nonzero(want) > want.size * nonzero_fraction
    return rel, rms


@pytest.mark.parametrize("T_,E,k", [(64, 32, 2), (300, 256, 8), (17, 64, 1)])
def test_route_topk(T_, E, k):
    from mosaicist_b200 import _lib

    logits = np.random.default_rng([T_, E]).standard_normal((T_, E)).astype(np.float32)
    ids = torch.empty((T_, k), dtype=torch.int32, device="cuda")
    w = torch.empty((T_, k), dtype=torch.float32, device="cuda")
    lt = T(logits)
    _lib.check(_lib.load().msc_moe_route_topk(lt.data_ptr(), ids.data_ptr(), w.data_ptr(), T_, E, k,
                                              torch.cuda.current_stream().cuda_stream))
    want_ids, want_w = M.route_topk(logits, k)
    assert np.array_equal(ids.cpu().numpy(), want_ids)
    assert np.allclose(w.cpu().numpy(), want_w, rtol=2e-6, atol=0)
    assert np.allclose(w.cpu().numpy().sum(1), 1.0, atol=1e-6)


def test_route_ties_go_to_lower_index():
    from mosaicist_b200 import _lib

    logits = np.zeros((4, 64), np.float32)
    logits[1, 40] = logits[1, 7] = 3.0
    ids = torch.empty((4, 3), dtype=torch.int32, device="cuda")
    w = torch.empty((4, 3), dtype=torch.float32, device="cuda")
    lt = T(logits)
    _lib.check(_lib.load().msc_moe_route_topk(lt.data_ptr(), ids.data_ptr(), w.data_ptr(), 4, 64, 3,
                                              torch.cuda.current_stream().cuda_stream))
    got = ids.cpu().numpy()
    assert got[0].tolist() == [0, 1, 2] and got[1].tolist() == [7, 40, 0]


@pytest.mark.parametrize("first,local,h,staged", [(0, 32, 256, False), (8, 8, 256, True), (0, 4, 320, False),
                                                  (0, 32, 768, True)])
def test_plan_and_gather_quantise_bit_exact(first, local, h, staged):
    """staged: the scale bytes leave as one bulk copy per row into a row-major buffer and a second
    kernel tiles them; otherwise they are written word by word.  Same bytes either way."""
    from mosaicist_b200 import _lib

    T_, E, k = 200, 32, 4
    rng = np.random.default_rng([first, local])
    logits = rng.standard_normal((T_, E)).astype(np.float32)
    logits[:, 5] = -30.0                              # an expert nobody picks: an empty group
    ids, w = M.route_topk(logits, k)
    tokens = rng.standard_normal((T_, h)).astype(np.float32).astype(ml_dtypes.bfloat16)
    gs = rng.uniform(200, 800, local).astype(np.float32)
    want_rank, want_rows, want_offs, want_tot = M.plan(ids, first, local)

    lib = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    d_ids, d_w = T(ids), T(w)
    rank = torch.full((T_, k), -7, dtype=torch.int32, device="cuda")
    rows = torch.zeros(local, dtype=torch.int32, device="cuda")
    offs = torch.zeros(local, dtype=torch.int32, device="cuda")
    tot = torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(4, dtype=torch.int32, device="cuda")
    for _ in range(2):                                # the ticket counter resets itself
        _lib.check(lib.msc_moe_plan(d_ids.data_ptr(), T_ * k, first, local, rank.data_ptr(),
                                    rows.data_ptr(), offs.data_ptr(), tot.data_ptr(),
                                    scratch.data_ptr(), st))
    assert int(scratch[0]) == 0
    assert np.array_equal(rows.cpu().numpy(), want_rows) and np.array_equal(offs.cpu().numpy(), want_offs)
    assert int(tot[0]) == want_tot
    local_mask = (ids >= first) & (ids < first + local)
    assert np.array_equal(rank.cpu().numpy()[local_mask], want_rank[local_mask])
    assert (rank.cpu().numpy()[~local_mask] == -7).all()

    cap = (T_ * k + 127 * local + 127) // 128 * 128
    a_q = torch.zeros((cap, h // 2), dtype=torch.uint8, device="cuda")
    a_sf = torch.zeros((cap // 128, h // 64, 32, 16), dtype=torch.uint8, device="cuda")
    rw = torch.zeros(cap, dtype=torch.float32, device="cuda")
    rt = torch.full((cap,), -1, dtype=torch.int32, device="cuda")
    tk = T(np.asarray(tokens, np.float32)).to(torch.bfloat16)
    gst = T(gs)
    sf_rows = torch.zeros((cap, h // 16), dtype=torch.uint8, device="cuda") if staged else None
    _lib.check(lib.msc_moe_permute_quantize(tk.data_ptr(), d_ids.data_ptr(), d_w.data_ptr(),
                                            rank.data_ptr(), offs.data_ptr(), gst.data_ptr(), T_, h, k,
                                            first, local, a_q.data_ptr(), a_sf.data_ptr(),
                                            rw.data_ptr(), rt.data_ptr(),
                                            sf_rows.data_ptr() if staged else None, cap,
                                            tot.data_ptr() if staged else None, st))
    qh, rth, rwh = a_q.cpu().numpy(), rt.cpu().numpy(), rw.cpu().numpy()
    sfh = np.asarray(__import__("mosaicist_b200.formats", fromlist=["x"]).from_mma_scale_layout(
        a_sf.cpu().numpy(), cap))
    seen = 0
    for t in range(T_):
        for kk in range(k):
            le = ids[t, kk] - first
            if not 0 <= le < local:
                continue
            row = want_offs[le] + want_rank[t, kk]
            q, sf = O.quantize_nvfp4(np.asarray(tokens[t:t + 1], np.float32)[None], gs[le:le + 1])
            assert np.array_equal(qh[row], O.pack_e2m1(q)[0, 0])
            assert np.array_equal(sfh[row], O.e4m3_bytes(sf)[0, 0])
            assert rth[row] == t and rwh[row] == w[t, kk]
            seen += 1
    assert seen == int(want_rows.sum()) and seen > 0 and (want_rows == 0).any() == (first <= 5 < first + local)


def test_unpermute_exact():
    from mosaicist_b200 import _lib

    T_, E, k, h = 100, 32, 4, 64
    rng = np.random.default_rng(3)
    ids, _ = M.route_topk(rng.standard_normal((T_, E)).astype(np.float32), k)
    rank, rows, offs, tot = M.plan(ids, 0, E)
    y = rng.integers(-8, 9, (tot, h)).astype(np.float32)       # exact in bf16, sums exact in fp32
    want = np.zeros((T_, h), np.float32)
    for t in range(T_):
        for kk in range(k):
            want[t] += y[offs[ids[t, kk]] + rank[t, kk]]
    out = torch.empty((T_, h), dtype=torch.bfloat16, device="cuda")
    yt = T(y).to(torch.bfloat16)
    di, dr, do = T(ids), T(rank), T(offs)
    _lib.check(_lib.load().msc_moe_unpermute(yt.data_ptr(), di.data_ptr(), dr.data_ptr(), do.data_ptr(),
                                             out.data_ptr(), T_, h, k, 0, E,
                                             torch.cuda.current_stream().cuda_stream))
    assert np.array_equal(out.float().cpu().numpy(), want)


# the two shapes of test_kernels.py:94-95, then the shape the reference times end to end
# (experiments/flashinfer-megamoe-sm100a/README.md:45-51)
@pytest.mark.parametrize("l,m,k,n", [(2, 256, 512, 256), (3, 128, 512, 512), (8, 512, 2048, 1024)])
def test_moe_masked_matches_reference_layer(l, m, k, n):
    from mosaicist_b200 import _lib
    from mosaicist_b200.moe import moe_masked

    w = _weights(l, k, n, seed=l)
    rng = np.random.default_rng([l, 1])
    hidden = rng.standard_normal((l, m, k)).astype(np.float32).astype(ml_dtypes.bfloat16)
    masked_m = np.array(([m, max(1, m // 2 - 3)] + [m] * l)[:l], np.int32)
    in_gs = O.global_scale_for(np.asarray(hidden, np.float32))
    a_q, a_sf = O.quantize_nvfp4(hidden, in_gs)
    gateup = O.masked_grouped_gemm_reference(a_q, a_sf, in_gs, w["w1_q"], w["w1_sf"], w["w1_gs"],
                                             w["w1_alpha"], masked_m)
    a2_gs = O.global_scale_for(O.silu_mul(gateup))               # moe.py:101-106
    want = np.asarray(O.moe_reference(hidden, w["w1_q"], w["w1_sf"], w["w1_gs"], w["w1_alpha"],
                                      w["w2_q"], w["w2_sf"], w["w2_gs"], w["w2_alpha"], masked_m,
                                      in_gs, a2_gs), np.float32)
    d = _dev_weights(w)
    args = (T(np.asarray(hidden, np.float32)).to(torch.bfloat16), d["w1_q"], d["w1_sf"],
            d["w1_gs"], d["w1_alpha"], d["w2_q"], d["w2_sf"], d["w2_gs"], d["w2_alpha"],
            T(masked_m), T(in_gs), T(a2_gs))
    from mosaicist_b200.moe import fold_alphas

    got = moe_masked(*args, fuse_gemm1=True)             # GEMM1 + SiLU*up + quantise in one kernel
    folded = fold_alphas(d["w1_gs"], d["w1_alpha"], d["w2_gs"], d["w2_alpha"], T(in_gs), T(a2_gs))
    three = moe_masked(*args, fuse_gemm1=False, folded_alphas=folded)     # the three-kernel form
    assert _lib.status_word() == 0
    rows = np.arange(m)[None, :, None] < masked_m[:, None, None]
    _close(np.where(rows, got.float().cpu().numpy(), 0), want)
    rows_t = torch.from_numpy(np.broadcast_to(rows, (l, m, k)).copy()).cuda()
    assert torch.equal(torch.where(rows_t, got, torch.zeros_like(got)),
                       torch.where(rows_t, three, torch.zeros_like(three)))
    # the layer as a torch operator: the same bits in the rows that count, zeros elsewhere
    import mosaicist_b200.torch_ops  # noqa: F401

    op = torch.ops.mosaicist_sm100a.moe_masked(*args)
    assert torch.equal(op, torch.where(rows_t, moe_masked(*args), torch.zeros_like(got)))


@pytest.mark.parametrize("form", ["f32", "scalar", "strided", "folded_only", "wide_w2", "no_alpha"])
@pytest.mark.parametrize("n", [256, 192])
def test_moe_masked_takes_every_form_its_steps_take(form, n):
    """The one-call layer reads bf16 activations and per-expert fp32 factors; fp32 activations, factors
    to broadcast or copy, folded factors alone and a second weight of another width take the separate
    steps, through the function and the torch operator alike."""
    import mosaicist_b200.torch_ops  # noqa: F401
    from mosaicist_b200 import _lib
    from mosaicist_b200.moe import fold_alphas, moe_masked

    l, m, k = 2, 128, 256
    d = _dev_weights(_weights(l, k, n, seed=n))
    rows = torch.tensor([128, 37], dtype=torch.int32, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(n)
    hidden = torch.randn((l, m, k), device="cuda", generator=gen).bfloat16()
    gs, a2 = torch.full((l,), 500.0, device="cuda"), torch.full((l,), 800.0, device="cuda")
    if form == "scalar":
        d["w1_alpha"], d["w2_gs"] = torch.full((l,), 0.75, device="cuda"), torch.full((l,), 300.0, device="cuda")
    w = [d[x] for x in ("w1_q", "w1_sf", "w1_gs", "w1_alpha", "w2_q", "w2_sf", "w2_gs", "w2_alpha")]
    live = torch.arange(m, device="cuda")[None, :, None] < rows[:, None, None]
    want = torch.where(live, moe_masked(hidden, *w, rows, gs, a2), 0)
    assert int((want != 0).sum()) > 0.9 * int(live.sum()) * k
    folded, operator = None, True
    if form == "f32":
        hidden = hidden.float()
    elif form == "scalar":
        w[3], w[6] = torch.tensor(0.75, device="cuda"), torch.tensor([300.0], device="cuda")
    elif form == "strided":
        w[2], w[7] = (torch.stack([x, torch.zeros_like(x)], 1)[:, 0] for x in (w[2], w[7]))
        assert not w[2].is_contiguous()
    elif form == "folded_only":
        folded, operator = fold_alphas(w[2], w[3], w[6], w[7], gs, a2), False
        w[2] = w[3] = w[6] = w[7] = None
    elif form == "wide_w2":
        w[4], w[5] = torch.cat([w[4], w[4]], 1).contiguous(), torch.cat([w[5], w[5]], 1).contiguous()
        want = torch.cat([want, want], 2)
    elif form == "no_alpha":            # a folded pair without the second factor: it counts as one
        first, second = fold_alphas(w[2], w[3], w[6], w[7], gs, a2)
        w[7] = torch.ones(l, device="cuda") * (a2 * w[6])
        want = torch.where(live, moe_masked(hidden, *w, rows, gs, a2, folded_alphas=(first, torch.ones_like(second))), 0)
        folded, operator = (first, None), False
    got = moe_masked(hidden, *w, rows, gs, a2, folded_alphas=folded)
    assert torch.equal(torch.where(live, got, 0), want)
    if operator:
        assert torch.equal(torch.ops.mosaicist_sm100a.moe_masked(hidden, *w, rows, gs, a2), want)
    assert _lib.status_word() == 0


@pytest.mark.parametrize("T_,E,k,h,n,first,local", [(256, 32, 4, 256, 128, 0, 32),
                                                     (384, 32, 2, 512, 256, 8, 8)])
def test_megamoe_layer(T_, E, k, h, n, first, local):
    from mosaicist_b200 import _lib
    from mosaicist_b200.moe import MegaMoE

    w = _weights(local, h, n, seed=T_)
    rng = np.random.default_rng([T_, 2])
    tokens = rng.standard_normal((T_, h)).astype(np.float32).astype(ml_dtypes.bfloat16)
    logits = rng.standard_normal((T_, E)).astype(np.float32)
    input_gs = np.full(local, 2688.0 / np.abs(np.asarray(tokens, np.float32)).max(), np.float32)
    a2_gs = np.full(local, 2688.0 / 4.0, np.float32)
    ids, wts = M.route_topk(logits, k)
    want = M.routed_moe(tokens, ids, wts, w["w1_q"], w["w1_sf"], w["w1_gs"], w["w1_alpha"], w["w2_q"],
                        w["w2_sf"], w["w2_gs"], w["w2_alpha"], input_gs, a2_gs, first)
    d = _dev_weights(w)
    layer = MegaMoE(d["w1_q"], d["w1_sf"], d["w1_gs"], d["w1_alpha"], d["w2_q"], d["w2_sf"], d["w2_gs"],
                    d["w2_alpha"], T(input_gs), T(a2_gs), topk=k, max_tokens=T_, expert_first=first)
    tk = T(np.asarray(tokens, np.float32)).to(torch.bfloat16)
    for _ in range(2):                                 # workspaces and the plan ticket are reusable
        got = layer.forward(tk, T(logits)).float().cpu().numpy()
    assert _lib.status_word() == 0
    assert np.array_equal(layer.ids.cpu().numpy(), ids)
    # with 8 of 32 experts local most tokens get no contribution: expect about 1 - (3/4)^2 non-zero
    _close(got, want, nonzero_fraction=0.5 if local == E else 0.25)
    # the layer's fused GEMM1 runs on the tokens-on-N kernel by default; on the row-major pair
    # kernel, and as separate GEMM + activation kernels, it produces the very same bits
    assert layer.gemm1_config.cta_pair == 3
    for kw in (dict(gemm1_tokens_on_n=False), dict(fuse_gemm1=False)):
        other = MegaMoE(d["w1_q"], d["w1_sf"], d["w1_gs"], d["w1_alpha"], d["w2_q"], d["w2_sf"], d["w2_gs"],
                        d["w2_alpha"], T(input_gs), T(a2_gs), topk=k, max_tokens=T_, expert_first=first, **kw)
        assert other.gemm1_config.cta_pair == 0
        assert np.array_equal(other.forward(tk, T(logits)).float().cpu().numpy(), got)
    assert _lib.status_word() == 0


@pytest.mark.parametrize("rows_list,n,k,swap", [([256], 128, 256, False), ([300, 0, 77, 512, 129], 256, 640, False),
                                                # tokens on the MMA's N side: one and two MMAs per tile,
                                                # several token tiles, every width of the narrow MMA
                                                ([256], 128, 256, True), ([300, 0, 77, 576, 129, 257, 320, 321, 16], 256, 640, True),
                                                ([272, 1, 240, 305], 512, 896, True)])
def test_fused_gemm1_swiglu_quantize_equals_two_kernel_path(rows_list, n, k, swap):
    """The fused epilogue must produce the very bytes of GEMM1 -> bf16 -> SiLU*up -> quantise;
    swap: the tokens-on-N kernel on the interleaved copy of w1."""
    from mosaicist_b200 import _lib, ops
    from mosaicist_b200.formats import from_mma_scale_layout

    l = len(rows_list)
    offs, tot = [], 0
    for r in rows_list:
        offs.append(tot)
        tot += (r + 127) // 128 * 128
    rng = np.random.default_rng([l, n, k])
    x = rng.standard_normal((1, tot, k)).astype(np.float32)
    a_q, a_sf = O.quantize_nvfp4(x, np.array([300.0], np.float32))
    w1 = (rng.standard_normal((l, 2 * n, k)) * 0.05).astype(np.float32)
    w1_gs = O.global_scale_for(w1)
    w1_q, w1_sf = O.quantize_nvfp4(w1, w1_gs)
    alpha = (rng.uniform(0.5, 1.5, l) / (300.0 * w1_gs)).astype(np.float32)
    a2_gs = rng.uniform(300, 900, l).astype(np.float32)
    dev = dict(a_q=T(O.pack_e2m1(a_q[0])), a_sf=T(O.e4m3_bytes(O.to_mma_scale_layout(a_sf[0]))),
               w1_q=T(O.pack_e2m1(w1_q)), w1_sf=T(O.e4m3_bytes(O.retile(w1_sf))))
    o_t, r_t = T(np.array(offs, np.int32)), T(np.array(rows_list, np.int32))
    gateup = ops.ragged_grouped_gemm_nvfp4(dev["a_q"], dev["a_sf"], dev["w1_q"], dev["w1_sf"], o_t, r_t, T(alpha))
    want_q, want_sf = ops.quantize_nvfp4_ragged(gateup, T(a2_gs), o_t, r_t, silu=True)
    if swap:
        wi_q, wi_sf = ops.swiglu_interleave_w1(dev["w1_q"], dev["w1_sf"])
        got_q, got_sf = ops.ragged_gemm1_swiglu_quantize(dev["a_q"], dev["a_sf"], wi_q, wi_sf, o_t, r_t, T(alpha),
                                                         T(a2_gs), ops.GemmConfig(cta_pair=3))
    else:
        got_q, got_sf = ops.ragged_gemm1_swiglu_quantize(dev["a_q"], dev["a_sf"], dev["w1_q"], dev["w1_sf"], o_t, r_t,
                                                         T(alpha), T(a2_gs))
    assert _lib.status_word() == 0
    wq, gq = want_q.cpu().numpy(), got_q.cpu().numpy()
    wsf = from_mma_scale_layout(want_sf.cpu().numpy(), tot)
    gsf = from_mma_scale_layout(got_sf.cpu().numpy(), tot)
    seen = 0
    for o, r in zip(offs, rows_list):
        assert np.array_equal(gq[o:o + r], wq[o:o + r]) and np.array_equal(gsf[o:o + r], wsf[o:o + r])
        seen += int(np.count_nonzero(wq[o:o + r]))
    assert seen > sum(rows_list) * n // 8
    # and the oracle agrees on the dequantised activation to within one e2m1 step per block
    g0 = next(i for i, r in enumerate(rows_list) if r)
    gu = O.masked_grouped_gemm_reference(a_q[:, offs[g0]:offs[g0] + rows_list[g0]], a_sf[:, offs[g0]:offs[g0] + rows_list[g0]],
                                         np.ones(1, np.float32), w1_q[g0:g0 + 1], w1_sf[g0:g0 + 1], np.ones(1, np.float32),
                                         alpha[g0:g0 + 1], [rows_list[g0]])
    oq, osf = O.quantize_nvfp4(O.silu_mul(gu), a2_gs[g0:g0 + 1])
    sl = slice(offs[g0], offs[g0] + rows_list[g0])
    assert np.mean(gq[sl] == O.pack_e2m1(oq)[0]) > 0.99


@pytest.mark.parametrize("rows_list,n,k", [([(i * 5) % 17 * (i % 2) for i in range(66)], 128, 640), ([128, 65, 0, 3], 256, 1152),
                                           ([160, 129, 1], 128, 896)])
def test_fused_gemm1_ring_depths_equal_two_kernel_path(rows_list, n, k):
    test_fused_gemm1_swiglu_quantize_equals_two_kernel_path(rows_list, n, k, True)


def test_megamoe_layer_replays_from_a_cuda_graph():
    """The whole routed layer is stream-ordered launches without host synchronisation or
    allocation (given `out`), so it captures into one CUDA graph; replays reproduce the eager
    result for new inputs written into the captured buffers."""
    from mosaicist_b200 import _lib
    from mosaicist_b200.moe import MegaMoE

    T_, E, k, h, n = 256, 32, 4, 512, 256
    w = _weights(E, h, n, seed=77)
    d = _dev_weights(w)
    gs_in, gs_a2 = T(np.full(E, 2688.0 / 5.0, np.float32)), T(np.full(E, 2688.0 / 4.0, np.float32))
    layer = MegaMoE(d["w1_q"], d["w1_sf"], d["w1_gs"], d["w1_alpha"], d["w2_q"], d["w2_sf"], d["w2_gs"],
                    d["w2_alpha"], gs_in, gs_a2, topk=k, max_tokens=T_)
    g = torch.Generator(device="cuda").manual_seed(5)
    tokens = torch.randn((T_, h), device="cuda", generator=g).bfloat16()
    logits = torch.randn((T_, E), device="cuda", generator=g)
    out = torch.empty((T_, h), dtype=torch.bfloat16, device="cuda")
    layer.forward(tokens, logits, out=out)                     # warm-up: tensor maps, attributes
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            layer.forward(tokens, logits, out=out)
    for seed in (6, 7):
        g.manual_seed(seed)
        tokens.copy_(torch.randn((T_, h), device="cuda", generator=g).bfloat16())
        logits.copy_(torch.randn((T_, E), device="cuda", generator=g))
        graph.replay()
        torch.cuda.synchronize()
        replayed = out.clone()
        eager = layer.forward(tokens, logits)
        assert torch.equal(replayed, eager) and int((eager != 0).sum()) > eager.numel() // 2
    assert _lib.status_word() == 0


@pytest.mark.parametrize("tokens_n", [1, 296, 297, 512, 520])   # wide and narrow CTAs; direct and staged scales (4096 rows)
def test_dispatch_and_combine_forms_agree(tokens_n):
    """Scales written directly and through the staging buffer are the same bytes in live rows, and a
    token's combined row does not depend on how many tokens (CTAs per token) the call has."""
    from mosaicist_b200 import _lib
    from mosaicist_b200.formats import from_mma_scale_layout
    from mosaicist_b200.moe import MegaMoE, _host_ops

    E, k, h, n = 32, 8, 4352, 128
    rng = torch.Generator(device="cuda").manual_seed(tokens_n)
    u8 = lambda *s: torch.randint(0, 256, s, dtype=torch.uint8, device="cuda", generator=rng)
    one = torch.ones((E,), device="cuda")
    sf1 = torch.full((E, 2 * n // 128, h // 64, 32, 16), 0x38, dtype=torch.uint8, device="cuda")     # e4m3 1.0
    sf2 = torch.full((E, h // 128, n // 64, 32, 16), 0x38, dtype=torch.uint8, device="cuda")
    layer = MegaMoE(u8(E, 2 * n, h // 2), sf1, one, one * 1e-3, u8(E, h, n // 2), sf2, one, one, one * 500, one * 50,
                    topk=k, max_tokens=tokens_n)
    x = torch.randn((tokens_n, h), device="cuda", generator=rng).bfloat16()
    logits = torch.randn((tokens_n, E), device="cuda", generator=rng)
    out = layer.forward(x, logits)
    want_q, want_sf = layer.a_q.clone(), layer.a_sf.clone()
    layer.a_q.fill_(0), layer.a_sf.fill_(0)
    assert layer.sf_rows is not None
    layer.sf_rows = None
    _host_ops.moe_dispatch(layer, x, None)
    live = torch.zeros((layer.rows_cap,), dtype=torch.bool)
    for o, r in zip(layer.group_offsets.tolist(), layer.group_rows.tolist()):
        live[o:o + r] = True
    assert int(live.sum()) == tokens_n * k
    assert torch.equal(layer.a_q.cpu()[live], want_q.cpu()[live])
    sf = [torch.from_numpy(from_mma_scale_layout(s.cpu().numpy(), layer.rows_cap).copy()) for s in (layer.a_sf, want_sf)]
    assert torch.equal(sf[0][live], sf[1][live])
    few = min(tokens_n, 16)
    assert torch.equal(_host_ops.moe_combine(layer, x[:few], None), out[:few])
    assert int((out != 0).sum()) > out.numel() // 2
    assert _lib.status_word() == 0
