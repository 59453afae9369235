"""GPU parity tests: the CUDA path (through the C ABI) against the CPU oracle.

Bars: bit-exact for codes, scale bytes, ids, counts, offsets, permutation; expert outputs
within max-abs error / max-abs reference <= 1e-2 of the FP32 oracle.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-2  # max|out - ref| / max|ref|, the tolerance the north star states


def _rel(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return float((a - b).abs().max() / b.abs().max().clamp_min(1e-30))


def _mods():
    import muse_moe_w4a16 as m
    from muse_moe_w4a16 import inputs, _lib
    from oracle import moe_oracle as orc
    return m, inputs, _lib, orc


def _adversarial_weights(H, I, E, dev, seed=3):
    """Random codes (all 16, sign bits included) and scale bytes covering zero, subnormal,
    normal and the largest finite E4M3 values."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    special = torch.tensor([0x00, 0x01, 0x07, 0x08, 0x38, 0x40, 0x7E, 0x30, 0x3F, 0x20], dtype=torch.uint8)

    def mk(rows, K):
        codes = torch.randint(0, 256, (E, rows, K // 2), generator=g, dtype=torch.uint8)
        sf = special[torch.randint(0, len(special), (E, rows, K // 16), generator=g)]
        return codes.to(dev), sf.to(dev)

    w13, w13_sf = mk(2 * I, H)
    w2, w2_sf = mk(H, I)
    return {"w13": w13, "w13_sf": w13_sf.view(torch.float8_e4m3fn), "w13_gs": torch.full((E,), 1e-3, device=dev),
            "w2": w2, "w2_sf": w2_sf.view(torch.float8_e4m3fn), "w2_gs": torch.full((E,), 1e-3, device=dev)}


def test_repack_is_lossless_and_decode_matches_oracle(cuda_dev):
    m, inputs, _lib, orc = _mods()
    H, I, E = 512, 256, 3
    w = _adversarial_weights(H, I, E, cuda_dev)
    st = m.prepare(w, max_tokens=8)
    back = m.export_weights(st)
    for k in ("w13", "w2"):
        assert torch.equal(back[k], w[k])
    for k in ("w13_sf", "w2_sf"):
        assert torch.equal(back[k], w[k].view(torch.uint8))
    dq13, dq2 = m.dequant_packed(st)
    torch.cuda.synchronize()
    for dq, c, s in ((dq13, w["w13"], w["w13_sf"]), (dq2, w["w2"], w["w2_sf"])):
        ref = orc.dequant(c.cpu().numpy(), s.view(torch.uint8).cpu().numpy())
        got = dq.float().cpu().numpy()
        assert np.array_equal(got, ref)  # e2m1 * e4m3 is exact in BF16


def test_decode_all_codes_times_all_scale_bytes(cuda_dev):
    """Known-answer sweep: 16 codes x 256 scale bytes (NaN bytes included)."""
    m, inputs, _lib, orc = _mods()
    H, I, E = 512, 256, 1
    # w13 rows: row r uses scale byte r % 256 everywhere; codes cycle through all 16
    codes = (torch.arange(H // 2) % 8).to(torch.uint8)
    codes = (2 * codes) | ((2 * codes + 1) << 4)          # nibble pairs (0,1),(2,3)...(14,15)
    w13 = codes.repeat(2 * I, 1).unsqueeze(0).contiguous()
    sf13 = (torch.arange(2 * I) % 256).to(torch.uint8).unsqueeze(1).repeat(1, H // 16).unsqueeze(0).contiguous()
    w2 = torch.zeros((1, H, I // 2), dtype=torch.uint8)
    sf2 = torch.zeros((1, H, I // 16), dtype=torch.uint8)
    w = {"w13": w13.to(cuda_dev), "w13_sf": sf13.to(cuda_dev), "w13_gs": torch.ones(1, device=cuda_dev),
         "w2": w2.to(cuda_dev), "w2_sf": sf2.to(cuda_dev), "w2_gs": torch.ones(1, device=cuda_dev)}
    st = m.prepare(w, max_tokens=8)
    dq13, _ = m.dequant_packed(st)
    got = dq13[0].float().cpu().numpy()
    ref = orc.dequant(w13[0].numpy(), sf13[0].numpy())
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert np.array_equal(got[ok], ref[ok])


@pytest.mark.parametrize("T,E,k,mode", [(1, 128, 8, "softmax_topk"), (37, 128, 8, "softmax_topk"),
                                        (64, 256, 8, "sigmoid_bias"), (5, 8, 2, "softmax_topk"),
                                        (300, 512, 16, "sigmoid_bias")])
def test_route_topk_bit_exact_ids(cuda_dev, T, E, k, mode):
    m, inputs, _lib, orc = _mods()
    lib = _lib.load()
    g = torch.Generator(device="cpu").manual_seed(T * 131 + E)
    logits = torch.randn((T, E), generator=g)
    logits[:, : E // 4] = logits[:, E // 4: E // 2][:, : E // 4]  # exact ties between experts
    bias = torch.randn((E,), generator=g) * 0.1 if mode == "sigmoid_bias" else None
    cfg = _lib.MskMoeCfg(hidden=512, inter=256, n_experts=E, local_start=0, local_count=min(E, 256), top_k=k,
                         routing_mode=m._MODES[mode], route_scale=0.1767766952966369, post_norm_eps=1e-8,
                         max_tokens=T)
    ld = logits.to(cuda_dev)
    bd = None if bias is None else bias.to(cuda_dev)
    ids = torch.empty((T, k), dtype=torch.int32, device=cuda_dev)
    tw = torch.empty((T, k), dtype=torch.float32, device=cuda_dev)
    _lib.check(lib.msk_moe_route(ctypes.byref(cfg), _lib.ptr(ld), _lib.ptr(bd), _lib.ptr(ids), _lib.ptr(tw), T,
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "route")
    torch.cuda.synchronize()
    rid, rw = orc.route_topk(logits, k, mode, bias)
    got = ids.cpu()
    if mode == "sigmoid_bias":
        # The score sigmoid(l * scale) + bias is evaluated by two exp implementations (device, host)
        # that may differ in the last bits. An id may therefore differ from the oracle's only where the
        # two candidates' scores are within 4 ulp of each other ("tie-risk"); anything else fails.
        sel = (torch.sigmoid(logits * 0.1767766952966369) + bias).numpy()
        a, b = got.numpy(), rid.numpy()
        rows, slots = np.nonzero(a != b)
        for r, c in zip(rows, slots):
            sa, sb = sel[r, a[r, c]], sel[r, b[r, c]]
            assert abs(float(sa) - float(sb)) <= 4 * float(np.spacing(np.float32(max(abs(sa), abs(sb))))), (r, c, sa, sb)
        assert len(set(rows.tolist())) <= max(1, T // 20)   # near-ties are rare on random logits
        same = torch.from_numpy(~np.isin(np.arange(T), rows))
        assert torch.allclose(tw.cpu()[same], rw[same], rtol=1e-5, atol=1e-7)
    else:
        assert torch.equal(got, rid)
        assert torch.allclose(tw.cpu(), rw, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("T,E,k,lo,nloc", [(1, 128, 8, 0, 128), (7, 128, 8, 0, 128), (256, 128, 8, 0, 128),
                                           (100, 256, 8, 64, 32), (8192, 128, 8, 0, 128), (33, 8, 2, 0, 8),
                                           (4097, 256, 8, 32, 32)])
def test_sort_bit_exact(cuda_dev, T, E, k, lo, nloc):
    m, inputs, _lib, orc = _mods()
    lib = _lib.load()
    g = torch.Generator(device="cpu").manual_seed(T + 7 * E)
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(min(T, 512))]).to(torch.int32)
    if T > 512:
        ids = ids.repeat((T + 511) // 512, 1)[:T].contiguous()
        ids = (ids + torch.arange(T, dtype=torch.int32).unsqueeze(1) * 5) % E
    ids[0, 0] = -1  # a dropped entry, as the decode layer's local-id convention produces
    cfg = _lib.MskMoeCfg(hidden=512, inter=256, n_experts=E, local_start=lo, local_count=nloc, top_k=k, max_tokens=T)
    d = ids.to(cuda_dev)
    cnt = torch.zeros(nloc, dtype=torch.int32, device=cuda_dev)
    off = torch.zeros(nloc + 1, dtype=torch.int32, device=cuda_dev)
    perm = torch.full((T * k,), -7, dtype=torch.int32, device=cuda_dev)
    inv = torch.full((T * k,), -7, dtype=torch.int32, device=cuda_dev)
    _lib.check(lib.msk_moe_sort(ctypes.byref(cfg), _lib.ptr(d), T, _lib.ptr(cnt), _lib.ptr(off), _lib.ptr(perm),
                                _lib.ptr(inv), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "sort")
    torch.cuda.synchronize()
    rc, ro, rp, ri = orc.sort_routes(ids.numpy(), lo, nloc)
    R = int(ro[-1])
    assert np.array_equal(cnt.cpu().numpy(), rc)
    assert np.array_equal(off.cpu().numpy(), ro)
    assert np.array_equal(perm.cpu().numpy()[:R], rp)
    assert np.array_equal(inv.cpu().numpy(), ri)


def _run_forward(m, inputs, orc, dev, H, I, E, k, T, seed, post_norm=False, logits_kind="normal", lo=0, nloc=None,
                 **prep):
    nloc = E if nloc is None else nloc
    w = inputs.make_weights(H, I, nloc, seed, dev, post_norm=post_norm)
    st = m.prepare(w, local_start=lo, n_experts=E, top_k=k, max_tokens=max(T, 1), **prep)
    g = torch.Generator(device=dev).manual_seed(seed + 99)
    x = torch.randn((T, H), generator=g, device=dev).to(torch.bfloat16)
    logits = inputs.make_logits(T, E, logits_kind, seed, dev)
    out, ids, tw = m.kernel_fn({"hidden_states": x, "router_logits": logits}, st, return_routing=True)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    ref, parts = orc.moe_forward(x, ids, tw, w, local_start=lo, return_parts=True)
    views = m.workspace_views(st, T)
    return out, ref, parts, views, st, (x, ids, tw, w)


def _check_forward(out, ref, parts, views):
    assert np.array_equal(views["cnt"].cpu().numpy(), parts["cnt"])
    assert np.array_equal(views["off"].cpu().numpy(), parts["off"])
    R = int(parts["off"][-1])
    assert np.array_equal(views["perm"].cpu().numpy()[:R], parts["perm"])
    assert np.array_equal(views["inv"].cpu().numpy(), parts["inv"])
    assert _rel(views["inter"], parts["inter"]) <= TOL
    assert _rel(views["y"], parts["y"]) <= TOL
    assert _rel(out, parts["out_fp32"]) <= TOL


def test_forward_tiny_config0(cuda_dev):
    """Config 0: H=512, I=256, E=8, top-2, T=4, router weight in the module."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 512, 256, 8, 2, 4
    w = inputs.make_weights(H, I, E, 0, cuda_dev)
    g = torch.Generator(device=cuda_dev).manual_seed(0)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    w["router"] = torch.randn((E, H), generator=g, device=cuda_dev) * 0.02
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    out, ids, tw = m.kernel_fn({"hidden_states": x}, st, return_routing=True)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    logits = orc.router_logits(x.cpu(), w["router"].cpu())
    rid, rw = orc.route_topk(logits, k)
    assert torch.equal(ids.cpu(), rid)
    assert torch.allclose(tw.cpu(), rw, rtol=1e-4, atol=1e-6)
    ref, parts = orc.moe_forward(x, ids, tw, w, return_parts=True)
    _check_forward(out, ref, parts, m.workspace_views(st, T))


@pytest.mark.parametrize("T,tile,path,post", [(1, 0, 0, False), (5, 16, 0, True), (5, 16, 1, False), (5, 16, 2, True),
                                              (40, 32, 1, False), (70, 64, 1, True), (300, 128, 1, False),
                                              (9, 16, 0, True), (9, 16, 1, True), (600, 0, 1, True), (300, 128, 1, True),
                                              (32, 16, 0, False), (32, 32, 2, True), (17, 32, 0, True), (32, 16, 1, True)])
def test_forward_small_shapes(cuda_dev, T, tile, path, post):
    """Every token tile and, for a few tokens, every path (0 one launch, 1 chain of launches, 2 row
    copy + routing gate/up kernel + combining down kernel)."""
    m, inputs, _lib, orc = _mods()
    out, ref, parts, views, st, _ = _run_forward(m, inputs, orc, cuda_dev, 512, 256, 8, 2, T, seed=T, post_norm=post,
                                                 token_tile=tile, decode_path=path or 3, flat_shares=1)
    if T <= 32:
        assert m.plan(st, T)[1] == path
    _check_forward(out, ref, parts, views)


@pytest.mark.parametrize("T,path,ctas,post", [(1, 0, 0, False), (1, 0, 37, True), (1, 2, 0, True), (1, 1, 0, False),
                                              (3, 0, 5, True), (3, 2, 148, False), (8, 0, 0, True), (8, 2, 37, False),
                                              (8, 1, 100, True), (32, 0, 0, True), (32, 0, 111, False), (32, 2, 0, True),
                                              (20, 0, 1, False), (2, 0, 148, True)])
def test_forward_few_token_paths_and_grids(cuda_dev, T, path, ctas, post):
    """Few tokens: the weight stream is cut into equal shares per CTA, so units are summed from pieces
    whose cut points move with the grid size; the kernels route, sort and combine themselves (paths 0
    and 2). Every combination must match the oracle, give the same bits with the routing passed in
    instead of the logits, and stay within rounding of the chain of launches."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 512, 16, 4
    out, ref, parts, views, st, (x, ids, tw, w) = _run_forward(m, inputs, orc, cuda_dev, H, I, E, k, T, seed=60 + T,
                                                               post_norm=post, decode_path=path or 3, num_ctas=ctas,
                                                               flat_shares=1)
    plan = m.plan(st, T)
    assert plan[1] == path and plan[2] == (0 if path == 0 else 1) and plan[3] == (ctas or 148)
    _check_forward(out, ref, parts, views)
    again = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, st)
    assert torch.equal(again, out)
    chain = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, decode_path=1, token_tile=16, num_ctas=3, flat_shares=1)
    other = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, chain)
    assert _rel(out, other) <= 8e-3   # same products, other cut points: a bf16 ulp or two of the output
    torch.cuda.synchronize()
    assert m.read_status(st) == 0 and m.read_status(chain) == 0


@pytest.mark.parametrize("T,H,I,E,k,lo,nloc,ctas,post,given", [
    (1, 256, 256, 4, 1, 0, 4, 0, False, False),        # one K block per GEMM, fewer row groups than CTAs
    (3, 768, 512, 300, 5, 7, 250, 0, True, False),     # odd number of K blocks, more experts than four per lane
    (2, 2304, 768, 16, 16, 0, 16, 11, True, False),    # widest top-k, several row groups per CTA
    (1, 7168, 2048, 8, 8, 0, 8, 0, False, False),      # 28 and 8 K blocks, four row groups per CTA
    (2, 1024, 512, 8, 16, 2, 4, 0, True, True),        # given ids that repeat an expert: tiles of 8 rows and a rest
    (3, 1024, 512, 8, 2, 6, 2, 37, False, True)])      # most routes elsewhere
def test_few_token_kernel_edges(cuda_dev, T, H, I, E, k, lo, nloc, ctas, post, given):
    """The one-launch kernel of up to three tokens at the edges of its units, teams, tiles and dealing of work,
    against the oracle, twice on one state (its counters are back at zero)."""
    m, inputs, _lib, orc = _mods()
    w = inputs.make_weights(H, I, nloc, 300 + T, cuda_dev, post_norm=post)
    st = m.prepare(w, local_start=lo, n_experts=E, top_k=k, max_tokens=T, num_ctas=ctas)
    g = torch.Generator(device=cuda_dev).manual_seed(700 + H)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    if given:
        d = {"topk_ids": torch.randint(-1, E, (T, k), generator=g, device=cuda_dev, dtype=torch.int32),
             "topk_weights": torch.rand((T, k), generator=g, device=cuda_dev)}
    else:
        d = {"router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    for _ in range(2):
        out, ids, tw = m.kernel_fn({"hidden_states": x, **d}, st, return_routing=True)
        torch.cuda.synchronize()
        assert m.read_status(st) == 0
        if not given:
            assert torch.equal(ids.cpu(), orc.route_topk(d["router_logits"].cpu(), k)[0])
        ref, parts = orc.moe_forward(x, ids, tw, w, local_start=lo, return_parts=True)
        _check_forward(out, ref, parts, m.workspace_views(st, T))


def test_forward_decode_shape_T1_and_T8(cuda_dev):
    """Config 1/2 shape with fewer experts resident (E=16 of the 4096 x 1536 experts)."""
    m, inputs, _lib, orc = _mods()
    for T, path in ((1, 0), (8, 0), (1, 2), (8, 2), (8, 1)):
        out, ref, parts, views, st, _ = _run_forward(m, inputs, orc, cuda_dev, 4096, 1536, 16, 8, T, seed=10 + T,
                                                     decode_path=path or 3, flat_shares=1)
        assert m.plan(st, T)[:3] == (16, path, 0 if path == 0 else 1)
        _check_forward(out, ref, parts, views)


def test_ep_combine_kernel_matches_rank_order_sum(cuda_dev):
    """msk_ep_combine against the same rank-order FP32 sum in torch (bit-exact: same order, same
    arithmetic); rows of ranks a token does not route to are never read."""
    from muse_moe_w4a16 import ep

    n, T, H, k, per = 4, 300, 512, 3, 8
    g = torch.Generator(device=cuda_dev).manual_seed(9)
    back = torch.randn((n, T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(n * per, generator=g, device=cuda_dev)[:k] for _ in range(T)]).to(torch.int32)
    ids[0] = -1  # a token with no route anywhere sums to zero
    mask = ep.route_mask(ids, n, per)
    poisoned = back.clone()
    poisoned[~mask] = float("nan")
    got = ep.combine_partials(poisoned, ids, per)
    want = ep.combine_partials(back.cpu(), ids.cpu(), per)
    assert torch.equal(got.cpu(), want)
    assert float(got[0].float().abs().max()) == 0.0
    own = ep.combine_partials(poisoned, ids, per, self_rank=1, self_rows=back[1].contiguous())
    assert torch.equal(own, got)


@pytest.mark.parametrize("tile,path", [(16, 0), (16, 1), (16, 2), (32, 0)])
def test_forward_local_range_negative_ids_and_empty_tokens(cuda_dev, tile, path):
    """Experts [4, 12) of 16 resident: routes outside the range and negative ids are dropped (the
    reference's filter, muse_moe_w4a16/cuda/moe.cu:347-350); a token left without any route is zero."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T, lo, nloc = 512, 256, 16, 4, 6, 4, 8
    w = inputs.make_weights(H, I, nloc, 31, cuda_dev, post_norm=True)
    st = m.prepare(w, local_start=lo, n_experts=E, top_k=k, max_tokens=T, token_tile=tile, decode_path=path or 3,
                   flat_shares=1)
    g = torch.Generator(device=cuda_dev).manual_seed(5)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    ids = torch.stack([torch.randperm(E, generator=g, device=cuda_dev)[:k] for _ in range(T)]).to(torch.int32)
    ids[1] = torch.tensor([0, 1, 14, 15], dtype=torch.int32)      # nothing local
    ids[2, 0] = -1
    ids[3] = -1                                                   # no route at all
    tw = torch.rand((T, k), generator=g, device=cuda_dev)
    out = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, st)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    ref, parts = orc.moe_forward(x, ids, tw, w, local_start=lo, return_parts=True)
    _check_forward(out, ref, parts, m.workspace_views(st, T))
    assert float(out[1].float().abs().max()) == 0.0 and float(out[3].float().abs().max()) == 0.0


@pytest.mark.parametrize("T", [1, 8, 40])
def test_forward_is_deterministic_and_graph_capturable(cuda_dev, T):
    """Same inputs, same bits: across calls, and between an eager call and a CUDA-graph replay."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 512, 16, 4
    w = inputs.make_weights(H, I, E, 41, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    g = torch.Generator(device=cuda_dev).manual_seed(6)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    first = m.kernel_fn(data, st).clone()
    for _ in range(3):
        assert torch.equal(m.kernel_fn(data, st), first)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        m.kernel_fn(data, st)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = m.kernel_fn(data, st)
    for _ in range(2):
        captured.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, first)
    assert m.read_status(st) == 0


def test_forward_zero_tokens_and_state_deepcopy(cuda_dev):
    import copy

    m, inputs, _lib, orc = _mods()
    H, I, E, k = 512, 256, 8, 2
    w = inputs.make_weights(H, I, E, 43, cuda_dev)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=4)
    empty = m.kernel_fn({"hidden_states": torch.empty((0, H), dtype=torch.bfloat16, device=cuda_dev),
                         "topk_ids": torch.empty((0, k), dtype=torch.int32, device=cuda_dev),
                         "topk_weights": torch.empty((0, k), device=cuda_dev)}, st)
    assert tuple(empty.shape) == (0, H)
    st2 = copy.deepcopy(st)
    g = torch.Generator(device=cuda_dev).manual_seed(8)
    data = {"hidden_states": torch.randn((3, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "router_logits": torch.randn((3, E), generator=g, device=cuda_dev)}
    assert torch.equal(m.kernel_fn(data, st), m.kernel_fn(data, st2))


@pytest.mark.parametrize("T,E,k,lo,nloc", [(8192, 8, 2, 0, 8), (4096, 16, 4, 4, 8)])
def test_forward_many_entries_sorted_on_several_ctas(cuda_dev, T, E, k, lo, nloc):
    """From 16384 routed entries on, the stable sort runs on several CTAs (count, scan, scatter); the
    tables must still equal the oracle's stable sort bit for bit, with and without a local range."""
    m, inputs, _lib, orc = _mods()
    out, ref, parts, views, st, _ = _run_forward(m, inputs, orc, cuda_dev, 512, 256, E, k, T, seed=77, post_norm=True,
                                                 lo=lo, nloc=nloc, logits_kind="zipf")
    assert T * k >= 16384
    _check_forward(out, ref, parts, views)


@pytest.mark.parametrize("T,E,k,lo,nloc", [(209, 300, 5, 20, 256),    # 27 CTAs, the last with one token; the most experts
                                           (520, 16, 16, 0, 16),      # 64 CTAs of nine tokens, the last ones without any
                                           (1024, 8, 1, 5, 2)])       # most routes elsewhere
def test_top_k_and_sort_on_several_ctas(cuda_dev, T, E, k, lo, nloc):
    """The top-k and the stable sort around the sizes from which they run on several CTAs (the second case does):
    tables equal to the oracle's. (The combine of the last case runs with few routes local.)"""
    m, inputs, _lib, orc = _mods()
    out, ref, parts, views, st, (x, ids, tw, w) = _run_forward(m, inputs, orc, cuda_dev, 256, 256, E, k, T, seed=79, lo=lo, nloc=nloc)
    rid, _ = orc.route_topk(inputs.make_logits(T, E, "normal", 79, cuda_dev).cpu(), k)
    assert torch.equal(ids.cpu(), rid)
    _check_forward(out, ref, parts, views)


@pytest.mark.parametrize("T,E,k,lo,nloc,several", [(425, 300, 5, 20, 256, True),     # 54 CTAs, the last with one token
                                                   (223, 128, 8, 0, 128, False), (224, 128, 8, 0, 128, True),   # 1784, 1792 local entries
                                                   (384, 256, 8, 64, 32, False),     # one rank of eight
                                                   (1535, 256, 8, 0, 8, False), (1536, 256, 8, 0, 8, True)])    # 12280, 12288 entries
def test_sort_moves_to_several_ctas_where_they_are_faster(cuda_dev, T, E, k, lo, nloc, several):
    """Few entries with a local expert are sorted by one CTA, many by several (whose counts are what the workspace
    then holds): the same tables as the oracle's either way, for logits and for the ids they gave."""
    m, inputs, _lib, orc = _mods()
    for given in (False, True):
        out, ref, parts, views, st, (x, ids, tw, w) = _run_forward(m, inputs, orc, cuda_dev, 256, 256, E, k, T, seed=83, lo=lo, nloc=nloc)
        if given:
            m.reinit_workspace(st)
            out = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, st)
            torch.cuda.synchronize()
            views = m.workspace_views(st, T)
        _check_forward(out, ref, parts, views)
        ptr = ctypes.c_void_p()
        _lib.check(st["lib"].lib.msk_moe_workspace_view(ctypes.byref(st["cfg"]), _lib.ptr(st["workspace"]), 9, ctypes.byref(ptr)),
                   "view")
        o = ptr.value - st["workspace"].data_ptr()
        assert bool(st["workspace"][o:o + 64 * 256 * 4].any()) == several


@pytest.mark.parametrize("T", [33, 64, 200])
def test_sort_reads_the_ids_of_the_top_k_in_front_of_it(cuda_dev, T):
    """Top-k and a sort on one CTA are two launches, the second there before the first has stored its ids: tables of back-to-back replays
    with other logits each time, each against its own ids."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 256, 256, 128, 8
    st = m.prepare(inputs.make_weights(H, I, E, 12, cuda_dev), n_experts=E, top_k=k, max_tokens=T)
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    many = torch.randn((12, T, E), generator=g, device=cuda_dev)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16), "router_logits": many[0].clone()}
    m.kernel_fn(data, st)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out, ids, tw = m.kernel_fn(data, st, return_routing=True)
    tables, ptr = [], ctypes.c_void_p()
    for which, n in ((0, E), (1, E + 1), (2, T * k), (3, T * k)):
        _lib.check(st["lib"].lib.msk_moe_workspace_view(ctypes.byref(st["cfg"]), _lib.ptr(st["workspace"]), which, ctypes.byref(ptr)), "view")
        at = ptr.value - st["workspace"].data_ptr()
        tables.append(st["workspace"][at:at + 4 * n].view(torch.int32))
    got = []
    for logits in many:
        data["router_logits"].copy_(logits)
        graph.replay()
        got.append([ids.clone()] + [t.clone() for t in tables])
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    for logits, (ids, *mine) in zip(many, got):
        rid, _ = orc.route_topk(logits.cpu(), k, "softmax_topk", None)
        assert torch.equal(ids.cpu(), rid)
        for a, b in zip(mine, orc.sort_routes(rid.numpy(), 0, E)):
            assert np.array_equal(a.cpu().numpy(), np.asarray(b).reshape(-1))


@pytest.mark.parametrize("tile,path,post,H,I", [(64, 0, False, 512, 256), (64, 1, True, 768, 512), (128, 0, True, 512, 256),
                                                (128, 0, False, 768, 512)])
def test_wide_tiles_at_ragged_row_counts(cuda_dev, tile, path, post, H, I):
    """The 64- and 128-token tiles around the heights of their activation boxes and the columns of their epilogue
    warps, the narrower one in one launch and in two, twice on one state; tokens with up to 12 routes for the combine."""
    m, inputs, _lib, orc = _mods()
    counts = [1, 15, 16, 17, 32, 33, 48, 0, 64, 65, 127, 128, 129]
    T, E = 131, len(counts)
    w = inputs.make_weights(H, I, E, 61, cuda_dev, post_norm=post)
    st = m.prepare(w, n_experts=E, top_k=E, max_tokens=T, token_tile=tile, decode_path=path)
    g = torch.Generator(device=cuda_dev).manual_seed(67)
    ids = torch.stack([torch.where(torch.randperm(T, generator=g, device=cuda_dev) < c, e, -1) for e, c in enumerate(counts)], 1)
    ids = ids.to(torch.int32).contiguous()
    tw = torch.rand((T, E), generator=g, device=cuda_dev)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    for _ in range(2):
        out = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, st)
        torch.cuda.synchronize()
        assert m.read_status(st) == 0
        ref, parts = orc.moe_forward(x, ids, tw, w, return_parts=True)
        _check_forward(out, ref, parts, m.workspace_views(st, T))


@pytest.mark.parametrize("H,I,ctas,post,nan", [(256, 256, 0, False, False), (512, 768, 2, True, False), (768, 256, 37, False, True),
                                               (1024, 512, 296, True, False), (512, 256, 1, False, False),
                                               (1536, 1280, 4, False, False)])
def test_pair_kernel_at_tile_edges(cuda_dev, H, I, ctas, post, nan):
    """The kernel on pairs of SMs around its tile heights (up to 256 rows an expert a tile, even shares of 32 beyond, one or both
    accumulator buffers), at its shortest reductions, with an odd grid, one pair and more CTAs than SMs; both GEMMs in one launch
    and in two give the same bits, twice on one state. A token of NaN leaves the rows of the others alone."""
    m, inputs, _lib, orc = _mods()
    counts = [1, 31, 32, 33, 64, 127, 128, 129, 160, 255, 256, 257, 300, 511, 513, 600]
    T, E = 600, len(counts)
    w = inputs.make_weights(H, I, E, 71, cuda_dev, post_norm=post)
    kw = dict(n_experts=E, top_k=E, max_tokens=T, token_tile=128, num_ctas=ctas)
    st, two = m.prepare(w, **kw), m.prepare(w, decode_path=1, **kw)
    g = torch.Generator(device=cuda_dev).manual_seed(73)
    ids = torch.stack([torch.where(torch.randperm(T, generator=g, device=cuda_dev) < c, e, -1) for e, c in enumerate(counts)], 1)
    ids = ids.to(torch.int32).contiguous()
    tw = torch.rand((T, E), generator=g, device=cuda_dev)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    data = {"hidden_states": x, "topk_ids": ids, "topk_weights": tw}
    ref, parts = orc.moe_forward(x, ids, tw, w, return_parts=True)
    for _ in range(2):
        out = m.kernel_fn(data, st)
        torch.cuda.synchronize()
        assert m.read_status(st) == 0
        _check_forward(out, ref, parts, m.workspace_views(st, T))
        assert torch.equal(m.kernel_fn(data, two), out)
        assert m.read_status(two) == 0
    if nan:
        bad = dict(data, hidden_states=x.clone())
        bad["hidden_states"][5] = float("nan")
        got = m.kernel_fn(bad, st)
        keep = torch.arange(T, device=cuda_dev) != 5
        assert torch.equal(got[keep], out[keep])


@pytest.mark.parametrize("H,I,ctas,counts", [(512, 768, 0, [64] * 8), (512, 768, 2, [100]), (1024, 1536, 0, [41, 128, 97, 64]),
                                             (1024, 1536, 2, [0, 90, 0]), (512, 4096, 0, [64, 65]), (512, 4096, 2, [128, 41, 77]),
                                             (2048, 1024, 0, [64] * 8), (2048, 1024, 37, [128] * 5 + [33]), (4096, 1536, 0, [64] * 6)])
def test_pair_kernel_hands_few_narrow_tiles_from_gate_up_to_down(cuda_dev, H, I, ctas, counts):
    """Few token tiles of one accumulator buffer and reductions of more A slots than the ring has: a cluster goes from its last gate/up
    unit straight to a down unit that may wait for it. Both GEMMs in one launch against two launches, bit for bit, and the oracle."""
    m, inputs, _lib, orc = _mods()
    E, T = len(counts), 128
    w = inputs.make_weights(H, I, E, 83, cuda_dev)
    kw = dict(n_experts=E, top_k=E, max_tokens=T, token_tile=128, num_ctas=ctas)
    st, two = m.prepare(w, **kw), m.prepare(w, decode_path=1, **kw)
    g = torch.Generator(device=cuda_dev).manual_seed(89)
    ids = torch.stack([torch.where(torch.randperm(T, generator=g, device=cuda_dev) < c, e, -1) for e, c in enumerate(counts)], 1)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "topk_ids": ids.to(torch.int32).contiguous(), "topk_weights": torch.rand((T, E), generator=g, device=cuda_dev)}
    ref, parts = orc.moe_forward(data["hidden_states"], data["topk_ids"], data["topk_weights"], w, return_parts=True)
    want = m.kernel_fn(data, two)
    assert m.read_status(two) == 0
    for _ in range(3):
        out = m.kernel_fn(data, st)
        assert m.read_status(st) == 0
        assert torch.equal(out, want)
    _check_forward(out, ref, parts, m.workspace_views(st, T))


@pytest.mark.parametrize("H,I,counts", [(256, 256, [8, 9, 15, 16, 17, 24, 47, 48]), (512, 768, [49, 79, 80, 81, 111, 112, 113, 144]),
                                        (768, 512, [145, 175, 176, 177, 209, 239, 240, 241])])
def test_pair_kernel_at_every_width_of_its_mmas(cuda_dev, H, I, counts):
    """MMAs are as wide as the tile's rows in steps of sixteen, half of them, eight at the least, in either CTA: rows around those
    steps, narrow and wide tiles in turn."""
    m, inputs, _lib, orc = _mods()
    E, T = len(counts), 256
    w = inputs.make_weights(H, I, E, 97, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=E, max_tokens=T, token_tile=128)
    g = torch.Generator(device=cuda_dev).manual_seed(101)
    ids = torch.stack([torch.where(torch.randperm(T, generator=g, device=cuda_dev) < c, e, -1) for e, c in enumerate(counts)], 1)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "topk_ids": ids.to(torch.int32).contiguous(), "topk_weights": torch.rand((T, E), generator=g, device=cuda_dev)}
    ref, parts = orc.moe_forward(data["hidden_states"], data["topk_ids"], data["topk_weights"], w, return_parts=True)
    out = m.kernel_fn(data, st)
    assert m.read_status(st) == 0
    _check_forward(out, ref, parts, m.workspace_views(st, T))


@pytest.mark.parametrize("H,T,k,tile,lo,nloc", [(4096, 255, 3, 16, 0, 12), (4096, 256, 9, 64, 0, 12), (4096, 256, 9, 128, 0, 12), (4352, 256, 3, 128, 4, 6),
                                                (8192, 257, 5, 128, 0, 12), (8192, 256, 5, 16, 0, 12), (8192, 255, 5, 128, 0, 12), (8192, 20, 9, 16, 2, 9),
                                                (256, 300, 16, 128, 0, 16), (256, 300, 2, 128, 3, 5)])
def test_combine_with_the_norm_at_its_block_sizes(cuda_dev, H, T, k, tile, lo, nloc):
    """The combine with the post-expert norm in each of its forms (few and many tokens, up to and beyond 4096 columns, FP32 and BF16
    rows, few and many local routes), tokens without a local route among them."""
    m, inputs, _lib, orc = _mods()
    E = 16 if nloc == 16 else 12
    w = inputs.make_weights(H, 256, nloc, 103, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, local_start=lo, token_tile=tile)
    g = torch.Generator(device=cuda_dev).manual_seed(107)
    ids = torch.rand((T, E), generator=g, device=cuda_dev).topk(k, 1)[1].to(torch.int32)
    ids[3] = ids[T - 1] = -1
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    tw = torch.rand((T, k), generator=g, device=cuda_dev)
    out = m.kernel_fn({"hidden_states": x, "topk_ids": ids.contiguous(), "topk_weights": tw}, st)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    assert not out[3].any() and not out[T - 1].any()
    ref, parts = orc.moe_forward(x, ids, tw, w, local_start=lo, return_parts=True)
    _check_forward(out, ref, parts, m.workspace_views(st, T))


@pytest.mark.parametrize("H,k,tile,lo,nloc", [(4096, 3, 16, 0, 12), (3840, 9, 64, 0, 12), (2048, 9, 64, 0, 12), (1024, 9, 128, 0, 12), (1536, 3, 128, 4, 6), (4096, 3, 128, 4, 6),
                                              (8192, 3, 16, 0, 12), (4352, 9, 128, 0, 12), (7168, 3, 128, 4, 6)])
def test_combine_with_the_norm_gives_a_token_the_same_bits_in_steps_of_any_size(cuda_dev, H, k, tile, lo, nloc):
    """The blocks of the combine with the post-expert norm are smaller from 256 tokens on: a row's squares are summed in the same order all the
    same, so that with one token tile a token's output does not change with the tokens beside it."""
    m, inputs, _lib, _ = _mods()
    E, T = 12, 257
    st = m.prepare(inputs.make_weights(H, 256, nloc, 109, cuda_dev, post_norm=True), n_experts=E, top_k=k, max_tokens=T, local_start=lo, token_tile=tile)
    g = torch.Generator(device=cuda_dev).manual_seed(113)
    ids = torch.rand((T, E), generator=g, device=cuda_dev).topk(k, 1)[1].to(torch.int32)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    tw = torch.rand((T, k), generator=g, device=cuda_dev)
    step = lambda n: m.kernel_fn({"hidden_states": x[:n], "topk_ids": ids[:n].contiguous(), "topk_weights": tw[:n].contiguous()}, st)  # noqa: E731
    most = step(T)
    for n in (9, 40, 255, 256):
        assert torch.equal(step(n), most[:n]), n
    assert m.read_status(st) == 0


@pytest.mark.parametrize("E,k,nloc,T", [(8, 2, 8, 256), (128, 8, 4, 700)])
def test_pair_kernel_by_default_on_a_handful_of_experts(cuda_dev, E, k, nloc, T):
    """The default plan takes the pair kernel by the mean rows per expert, also where only a handful of experts is there."""
    m, inputs, _lib, orc = _mods()
    H, I = 1024, 1536
    w = inputs.make_weights(H, I, nloc, 97, cuda_dev)
    st = m.prepare(w, n_experts=E, top_k=k, local_start=E // 2 - nloc // 2 if nloc < E else 0, max_tokens=T)
    assert m.plan(st, T)[0] == 128
    data = dict(hidden_states=torch.randn((T, H), device=cuda_dev, generator=torch.Generator(device=cuda_dev).manual_seed(5)).to(torch.bfloat16))
    ids = torch.stack([(torch.arange(T, device=cuda_dev) * k + j) % E for j in range(k)], 1).to(torch.int32)   # even rows
    tw = torch.full((T, k), 1.0 / k, device=cuda_dev)
    data.update(topk_ids=ids.contiguous(), topk_weights=tw)
    for _ in range(2):
        out = m.kernel_fn(data, st)
        assert m.read_status(st) == 0
    ref, parts = orc.moe_forward(data["hidden_states"], ids, tw, w, local_start=E // 2 - nloc // 2 if nloc < E else 0, return_parts=True)
    _check_forward(out, ref, parts, m.workspace_views(st, T))


@pytest.mark.parametrize("T,scale", [(131, 1.0), (700, 1.0), (300, 60.0)])
def test_every_token_tile_gives_the_same_swiglu_values(cuda_dev, T, scale):
    """inter of the 16-, 64- and 128-token tiles, bit for bit: the accumulators sum in the same order and the SwiGLU value
    is one formula (exactly rounded quotient included), whatever the epilogue. The last case takes gates to where the
    exponential over- and underflows."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 768, 512, 6, 3
    w = inputs.make_weights(H, I, E, 91, cuda_dev)
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    x = (torch.randn((T, H), generator=g, device=cuda_dev) * scale).to(torch.bfloat16)
    logits = torch.randn((T, E), generator=g, device=cuda_dev)
    got = {}
    for tile in (16, 64, 128):
        st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, token_tile=tile)
        m.kernel_fn({"hidden_states": x, "router_logits": logits}, st)
        torch.cuda.synchronize()
        assert m.read_status(st) == 0
        got[tile] = m.workspace_views(st, T)["inter"]
    assert torch.isfinite(got[16]).all() and float(got[16].abs().max()) > 0
    assert torch.equal(got[64], got[16]) and torch.equal(got[128], got[16])


def test_graphed_step_with_pinned_host_inputs(cuda_dev):
    """GraphedStep (static buffers + CUDA graph) returns what kernel_fn returns, bit for bit, for
    device inputs and for pinned host inputs, call after call."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 1024, 512, 16, 4, 5
    w = inputs.make_weights(H, I, E, 51, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    g = torch.Generator(device=cuda_dev).manual_seed(9)
    datas = [{"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
              "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)} for _ in range(3)]
    step = m.GraphedStep(st, datas[0])
    for d in datas + datas[:1]:
        want = m.kernel_fn(d, st)
        host = {key: v.cpu().pin_memory() for key, v in d.items()}
        got_dev = step(d).clone()
        got_host = step(host).clone()
        torch.cuda.synchronize()
        assert torch.equal(got_dev, want) and torch.equal(got_host, want)
    assert m.read_status(st) == 0


def test_graphed_step_runs_one_plan_for_all_inputs(cuda_dev):
    """A change of the state's configuration after the capture (okc_set_pdl, a forced tile) reaches neither the replays nor
    the calls launched on device tensors: both give the bits of the captured plan."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 512, 256, 8, 2, 40
    st = m.prepare(inputs.make_weights(H, I, E, 58, cuda_dev), n_experts=E, top_k=k, max_tokens=T, token_tile=16)
    g = torch.Generator(device=cuda_dev).manual_seed(11)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    want = m.kernel_fn(data, st).clone()
    step = m.GraphedStep(st, data)
    st["cfg"].token_tile = 128                        # keeps y in BF16: other bits
    assert not torch.equal(m.kernel_fn(data, st), want)
    assert torch.equal(step({key: v.cpu() for key, v in data.items()}), want)
    assert torch.equal(step(data), want)


@pytest.mark.parametrize("T,routed", [(2, False), (5, True), (40, True)])
def test_graphed_step_copies_device_tensors_the_kernels_cannot_read(cuda_dev, T, routed):
    """Device inputs of another type, off their alignment, strided, or some of them on the host are copied into the
    captured buffers and the graph is replayed: the bits of kernel_fn on the plain tensors, call after call."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 512, 256, 8, 2
    st = m.prepare(inputs.make_weights(H, I, E, 59, cuda_dev, post_norm=True), n_experts=E, top_k=k, max_tokens=T)
    g = torch.Generator(device=cuda_dev).manual_seed(13 + T)

    def draw():
        d = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)}
        logits = torch.randn((T, E), generator=g, device=cuda_dev).to(torch.bfloat16).float()
        if routed:
            tw, ids = torch.softmax(logits, dim=-1).topk(k, dim=-1)
            d["topk_ids"], d["topk_weights"] = ids.to(torch.int32).contiguous(), tw.contiguous()
        else:
            d["router_logits"] = logits
        return d

    def misaligned(t):
        flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
        return flat.view(t.shape).copy_(t)

    def strided(t):
        return torch.stack([t, t], -1)[..., 0]

    step = m.GraphedStep(st, draw())
    second = "topk_weights" if routed else "router_logits"
    for form in ("plain", "misaligned", "strided", "type", "host"):
        d = draw()
        want = m.kernel_fn(d, st).clone()
        e = dict(d)
        if form in ("misaligned", "strided"):
            e = {key: (misaligned if form == "misaligned" else strided)(v) for key, v in d.items()}
            assert not step._usable(e)
        elif form == "type":
            key = "topk_ids" if routed else "router_logits"
            e[key] = d[key].long() if routed else d[key].to(torch.bfloat16)      # (values of both survive the change)
            assert not step._usable(e)
        elif form == "host":
            e[second] = d[second].cpu()
        got = step(e)
        torch.cuda.synchronize()
        assert torch.equal(got, want), form
    assert m.read_status(st) == 0


@pytest.mark.parametrize("T,routed,I", [(1, False, 512), (5, False, 512), (8, True, 512), (40, False, 512),
                                        (4, False, 1536), (6, True, 1536), (8, False, 1536), (40, True, 1536)])     # the FP4 kernel
def test_host_mapped_step_reads_and_writes_pinned_host_memory(cuda_dev, T, routed, I):
    """HostMappedStep (kernels read the inputs from, and write the output to, pinned host memory; no copy
    launches) returns what kernel_fn returns on device tensors, bit for bit, call after call and across
    its ring of blocks: one-launch path (1, 5, 8 tokens), chain (40 tokens), given ids and logits; the FP4 kernel."""
    m, inputs, _lib, orc = _mods()
    H, E, k = 1024, 16, 4
    w = inputs.make_weights(H, I, E, 52, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    assert _nvf4_takes(st, T) == (I == 1536)
    g = torch.Generator(device=cuda_dev).manual_seed(10 + T)
    datas = []
    for _ in range(6):
        d = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)}
        logits = torch.randn((T, E), generator=g, device=cuda_dev)
        if routed:
            tw, ids = torch.softmax(logits, dim=-1).topk(k, dim=-1)
            d["topk_ids"], d["topk_weights"] = ids.to(torch.int32), tw.contiguous()
        else:
            d["router_logits"] = logits
        datas.append(d)
    step = m.HostMappedStep(st, {key: v.cpu() for key, v in datas[0].items()})
    for d in datas:
        want = m.kernel_fn(d, st)
        got = step({key: v.cpu() for key, v in d.items()})
        assert not got.is_cuda and got.is_pinned()
        step.done.synchronize()
        assert torch.equal(got, want.cpu())
    assert m.read_status(st) == 0


@pytest.mark.parametrize("T", [3, 4, 8])
@pytest.mark.parametrize("pre,ids", [(False, False), (True, False), (False, True)])
def test_few_tokens_with_the_post_norm_around_the_end_of_the_one_launch(cuda_dev, T, pre, ids):
    """Default steps on both sides of the line from which the post-expert norm takes launches of its own, against the oracle; from
    the line on with the bits of that form when it is asked for."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 512, 40, 5
    w = inputs.make_weights(H, I, E, 64, cuda_dev, post_norm=True)
    g = torch.Generator(device=cuda_dev).manual_seed(40 + T)
    if pre:
        w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=8)
    asked = m.prepare(w, n_experts=E, top_k=k, max_tokens=8, decode_path=4)
    data = {"hidden_states": (torch.randn((T, H), generator=g, device=cuda_dev) * 3.0).to(torch.bfloat16)}
    lg = torch.randn((T, E), generator=g, device=cuda_dev)
    if ids:
        tw, top = torch.softmax(lg, dim=-1).topk(k, dim=-1)
        data["topk_ids"], data["topk_weights"] = top.to(torch.int32).contiguous(), tw.contiguous()
    else:
        data["router_logits"] = lg
    form = m.step_form(st, T, given_ids=ids)
    assert form == ("few-token kernel" if T == 3 or (pre and T == 4) else "chain" if pre else "both GEMMs")
    for _ in range(2):
        same = m.kernel_fn(data, asked)
        got, top, tw = m.kernel_fn(data, st, return_routing=True)
        ref, parts = orc.moe_forward(data["hidden_states"], top, tw, w, return_parts=True)
        _check_forward(got, ref, parts, m.workspace_views(st, T))
        assert torch.equal(got, same) if form != "few-token kernel" else _rel(got, same.float()) <= TOL
        if not ids:
            assert torch.equal(top.cpu(), orc.route_topk(lg.cpu(), k)[0])
    if pre:      # the norm is not a no-op here
        assert _rel(got, orc.moe_forward(data["hidden_states"], top, tw, {n: v for n, v in w.items() if n != "pre_norm_w"}).float()) > 0.05
    assert m.read_status(st) == 0 and m.read_status(asked) == 0


@pytest.mark.parametrize("T,routed", [(4, False), (7, True), (8, False)])
def test_host_mapped_steps_of_a_few_tokens_without_a_norm(cuda_dev, T, routed):
    """Steps from pinned memory that the few-token kernel leaves take launches of their own where those on device tensors take one:
    the same units and the same order of sums, so the same bits."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 512, 40, 5
    w = inputs.make_weights(H, I, E, 65, cuda_dev, post_norm=False)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=8)
    g = torch.Generator(device=cuda_dev).manual_seed(50 + T)
    step = None
    for _ in range(3):
        d = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)}
        lg = torch.randn((T, E), generator=g, device=cuda_dev)
        if routed:
            tw, ids = torch.softmax(lg, dim=-1).topk(k, dim=-1)
            d["topk_ids"], d["topk_weights"] = ids.to(torch.int32), tw.contiguous()
        else:
            d["router_logits"] = lg
        host = {key: v.cpu() for key, v in d.items()}
        step = step or m.HostMappedStep(st, host)
        want, got = m.kernel_fn(d, st), step(host)
        step.done.synchronize()
        assert torch.equal(got, want.cpu())
    assert m.read_status(st) == 0


@pytest.mark.parametrize("T,E,k,nloc,H,host", [(1, 16, 8, 16, 256, "xl"), (2, 128, 8, 128, 1024, "xl"), (3, 130, 5, 130, 768, "xl"), (1, 512, 4, 256, 512, "xl"),
                                               (3, 512, 2, 40, 768, "xl"), (2, 16, 4, 16, 1024, "x"), (2, 16, 4, 16, 1024, "l"),
                                               (1, 16, 8, 16, 256, "xi"), (3, 130, 5, 130, 768, "xi"), (2, 512, 7, 40, 512, "xi"), (2, 16, 4, 16, 1024, "i")])
def test_routes_in_host_memory_are_fetched_once_for_all_ctas(cuda_dev, T, E, k, nloc, H, host):
    """The few-token kernel with its rows and logits, or given ids and weights, in pinned memory, one of them, both: routing and output are those on device
    tensors, bit for bit, from call to call (1 to 3 rows, rows that no warp's 32 lanes divide, the most experts, few of them local)."""
    m, inputs, _lib, orc = _mods()
    w = inputs.make_weights(H, 256, nloc, 63, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=4)
    g = torch.Generator(device=cuda_dev).manual_seed(30 + T)

    def run(x, logits=None, ids=None, tw=None):
        out = torch.empty((T, H), dtype=torch.bfloat16, device=cuda_dev)
        if ids is None:
            ids, tw = torch.empty((T, k), dtype=torch.int32, device=cuda_dev), torch.empty((T, k), device=cuda_dev)
        m._forward(st, st["cfg"], st["lib"].lib, x.data_ptr(), None if logits is None else logits.data_ptr(), ids.data_ptr(), tw.data_ptr(),
                   out.data_ptr(), T)
        torch.cuda.synchronize()
        return out, ids, tw

    for _ in range(3):
        x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
        logits = torch.randn((T, E), generator=g, device=cuda_dev)
        want = run(x, logits)
        xh = x.cpu().pin_memory() if "x" in host else x
        if "i" in host:
            got = run(xh, None, want[1].cpu().pin_memory(), want[2].cpu().pin_memory())
            assert torch.equal(got[0], want[0])
        else:
            got = run(xh, logits.cpu().pin_memory() if "l" in host else logits)
            assert all(torch.equal(u, v) for u, v in zip(got, want))
    assert m.read_status(st) == 0


@pytest.mark.parametrize("T,pre", [(1, False), (2, False), (1, True), (3, True)])
def test_pinned_token_rows_through_the_c_interface(cuda_dev, T, pre):
    """A host hands msk_moe_forward* pinned token rows and nothing else that says so: the CTAs share one F16 copy of them
    (it stands in the workspace afterwards), normed ones are read by another kernel, and the output is the one on device tensors."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 512, 16, 4
    w = inputs.make_weights(H, I, E, 53, cuda_dev, post_norm=True)
    g = torch.Generator(device=cuda_dev).manual_seed(20 + T)
    if pre:
        w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=8)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    tw, ids = torch.softmax(torch.randn((T, E), generator=g, device=cuda_dev), dim=-1).topk(k, dim=-1)
    ids, tw = ids.to(torch.int32).contiguous(), tw.contiguous()
    want = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, st)
    st["workspace"].zero_()
    xh, out = x.cpu().pin_memory(), torch.empty((T, H), dtype=torch.bfloat16, device=cuda_dev)
    m._forward(st, st["cfg"], st["lib"].lib, xh.data_ptr(), None, ids.data_ptr(), tw.data_ptr(), out.data_ptr(), T)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    if pre:
        assert _rel(out, want.float()) <= 8e-3      # two kernels, sums in another order: one BF16 rounding
    else:
        assert torch.equal(out, want)
        row = x[T - 1].to(torch.float16).view(torch.int64)
        words = st["workspace"].view(torch.int64)
        at = (words == row[0]).nonzero().flatten()
        assert any(torch.equal(words[int(a):int(a) + row.numel()], row) for a in at)


@pytest.mark.parametrize("T,nloc,host,post", [(2, 16, "x", False), (8, 16, "x", True), (3, 16, "xr", False), (8, 16, "xr", True), (8, 8, "xr", True),
                                              (8, 4, "", True), (8, 16, "", True), (7, 16, "r", True)])
@pytest.mark.parametrize("given", [False, True])
def test_few_tokens_with_the_pre_norm_in_the_chain_and_folded(cuda_dev, T, nloc, host, post, given):
    """Rows (x) and routes (r) on the device or in pinned memory, few and many local routes: both forms that steps with the pre-expert norm
    take beyond the few-token kernel, against the oracle, tables and routing included, twice on one state."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, lo = 1280, 512, 16, 4, 16 - nloc
    w = inputs.make_weights(H, I, nloc, 57, cuda_dev, post_norm=post)
    g = torch.Generator(device=cuda_dev).manual_seed(60 + T)
    w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=8, local_start=lo)
    place = lambda t, what: t.cpu().pin_memory() if what in host else t  # noqa: E731
    forms = set()
    for _ in range(2):
        x = (torch.randn((T, H), generator=g, device=cuda_dev) * 3.0).to(torch.bfloat16)
        lg = torch.randn((T, E), generator=g, device=cuda_dev)
        rid, _ = orc.route_topk(lg.cpu(), k)
        tw, ids = torch.empty((T, k), device=cuda_dev), torch.empty((T, k), dtype=torch.int32, device=cuda_dev)
        if given:
            tw, ids = torch.softmax(lg, dim=-1).topk(k, dim=-1)
            ids, tw = place(ids.to(torch.int32).contiguous(), "r"), place(tw.contiguous(), "r")
        xp, lp = place(x, "x"), None if given else place(lg, "r")
        out = torch.empty((T, H), dtype=torch.bfloat16, device=cuda_dev)
        m._forward(st, st["cfg"], st["lib"].lib, xp.data_ptr(), None if given else lp.data_ptr(), ids.data_ptr(), tw.data_ptr(), out.data_ptr(), T)
        torch.cuda.synchronize()
        assert m.read_status(st) == 0 and torch.equal(ids.cpu(), rid)
        ref, parts = orc.moe_forward(x, ids.to(cuda_dev), tw.to(cuda_dev), w, local_start=lo, return_parts=True)
        _check_forward(out, ref, parts, m.workspace_views(st, T))
        form = ctypes.c_int(0)
        bits = int(given) + 2 + 4 * ("x" in host) + 8 * post + 16 * (host == "xr")
        assert st["lib"].lib.msk_moe_step_form(ctypes.byref(st["cfg"]), T, bits, ctypes.byref(form)) == 0
        forms.add(form.value)
    assert forms == {1 if nloc == 16 and host != "x" else 2}


@pytest.mark.parametrize("T,tile", [(9, 0), (40, 0), (100, 16), (100, 32), (260, 32)])
def test_both_gemms_in_one_launch_behind_the_sort_gives_the_chain_bits(cuda_dev, T, tile):
    """decode_path = 4 (sort launches, then the gate/up and the down GEMM in one cooperative launch that
    hands `inter` over tile by tile, then the combine) computes every unit exactly as the chain of
    launches does: same output bits, same sort tables, status word clean, call after call."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 512, 16, 4
    w = inputs.make_weights(H, I, E, 53, cuda_dev, post_norm=True)
    chain = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, decode_path=1, token_tile=tile)
    both = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, decode_path=4, token_tile=tile)
    assert m.plan(both, T)[1] == 4 and m.plan(chain, T)[1] == 1
    g = torch.Generator(device=cuda_dev).manual_seed(20 + T)
    for _ in range(3):
        d = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
             "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
        want, ids_w, tw_w = m.kernel_fn(d, chain, return_routing=True)
        got, ids_g, tw_g = m.kernel_fn(d, both, return_routing=True)
        torch.cuda.synchronize()
        assert torch.equal(ids_g, ids_w) and torch.equal(tw_g, tw_w)
        assert torch.equal(got, want)
        vw, vg = m.workspace_views(chain, T), m.workspace_views(both, T)
        for key in ("cnt", "off", "perm", "inv"):
            assert torch.equal(vg[key], vw[key]), key
    assert m.read_status(both) == 0 and m.read_status(chain) == 0


def test_okc_ext_runs_the_decode_layer_call_site(cuda_dev):
    """The decode layer's call (muse_decode_layer/py/06_kernel_fn.py:140-149): local ids with -1 for
    another GPU's expert, lo = 0, an output slice filled in place, in chunks."""
    m, inputs, _lib, orc = _mods()
    from muse_moe_w4a16.compat import OkcExt

    H, I, nloc, k, T = 1024, 512, 8, 4, 11
    w = inputs.make_weights(H, I, nloc, 61, cuda_dev, post_norm=True)
    st = m.prepare(w, local_start=0, n_experts=nloc, top_k=k, max_tokens=8)
    ext = OkcExt(st)
    g = torch.Generator(device=cuda_dev).manual_seed(4)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    lids = torch.randint(-1, nloc, (T, k), generator=g, device=cuda_dev, dtype=torch.int32)
    wts = torch.rand((T, k), generator=g, device=cuda_dev)
    out = torch.full((T, H), float("nan"), dtype=torch.bfloat16, device=cuda_dev)
    ext.okc_set_pdl(1)
    for m0 in range(0, T, 8):
        m1 = min(T, m0 + 8)
        ext.okc_run(None, None, x[m0:m1], lids[m0:m1], wts[m0:m1], out[m0:m1], 0, nloc, 148)
    torch.cuda.synchronize()
    ref = orc.moe_forward(x, lids, wts, w).float()
    assert _rel(out, ref) <= TOL
    assert len(ext.okc_attrs()) == 6
    with pytest.raises(RuntimeError):
        ext.okc_run(None, None, x[:1], lids[:1], wts[:1], out[:1], 1, nloc, 148)
    with pytest.raises(RuntimeError):
        ext.okc_run(None, None, x[:1], lids[:1], wts[:1], out[:1], 0, nloc, 132)   # a grid it was not prepared for
    # without programmatic dependent launch the chain of launches gives the same bits
    ext.okc_set_pdl(0)
    out2 = torch.empty_like(out)
    for m0 in range(0, T, 8):
        m1 = min(T, m0 + 8)
        ext.okc_run(None, None, x[m0:m1], lids[m0:m1], wts[m0:m1], out2[m0:m1], 0, nloc, 148)
    torch.cuda.synchronize()
    assert torch.equal(out2, out)


def _programmatic_edges(graph):
    """Dependencies of a captured graph that are programmatic launches (driver API, CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC)."""
    driver, n = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t(0)
    raw = ctypes.c_void_p(graph.raw_cuda_graph())
    assert driver.cuGraphGetEdges_v2(raw, None, None, None, ctypes.byref(n)) == 0
    if n.value == 0:
        return 0
    src, dst, data = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (ctypes.c_ubyte * (8 * n.value))()
    assert driver.cuGraphGetEdges_v2(raw, src, dst, data, ctypes.byref(n)) == 0
    return sum(1 for i in range(n.value) if data[8 * i + 2] == 1)


@pytest.mark.parametrize("T,tile", [(24, 16), (40, 16), (300, 64), (300, 128)])     # one CTA sorts, routes apart, several CTAs
def test_no_step_is_chained_programmatically_when_that_is_switched_off(cuda_dev, T, tile):
    """okc_set_pdl(0) / cfg.no_pdl: every launch of a step that computes its logits, routes and sorts waits for the
    whole launch before it; with the switch on some of them do not. Same bits."""
    from muse_moe_w4a16 import compat

    m, inputs, _lib, orc = _mods()
    H, I, E, k = 512, 256, 16, 8
    w = inputs.make_weights(H, I, E, 57, cuda_dev)
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    w["router"] = torch.randn((E, H), generator=g, device=cuda_dev) * 0.02
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, token_tile=tile)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)}
    outs = []
    for on in (1, 0):
        compat.OkcExt(st).okc_set_pdl(on)
        m.kernel_fn(data, st)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            out = m.kernel_fn(data, st)
        assert (_programmatic_edges(graph) > 0) == bool(on)
        graph.instantiate()
        graph.replay()
        torch.cuda.synchronize()
        outs.append(out)
    assert m.read_status(st) == 0 and torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("T,given_ids", [(3, False), (7, True), (40, True), (300, False), (600, True)])
def test_forward_with_pre_expert_norm(cuda_dev, T, given_ids):
    """weights["pre_norm_w"]: the layer callers' pre-expert RMS norm (eps 1e-5, x (1 + g)) fused into
    the row-copy kernel, for every token-tile width; routing still sees the un-normed logits."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 512, 8, 2
    w = inputs.make_weights(H, I, E, 71, cuda_dev, post_norm=True)
    g = torch.Generator(device=cuda_dev).manual_seed(12)
    w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    x = (torch.randn((T, H), generator=g, device=cuda_dev) * 3.0).to(torch.bfloat16)
    logits = torch.randn((T, E), generator=g, device=cuda_dev)
    out, ids, tw = m.kernel_fn({"hidden_states": x, "router_logits": logits}, st, return_routing=True)
    if given_ids:
        out = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, st)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    rid, _ = orc.route_topk(logits.cpu(), k)
    assert torch.equal(ids.cpu(), rid)
    ref, parts = orc.moe_forward(x, ids, tw, w, return_parts=True)
    _check_forward(out, ref, parts, m.workspace_views(st, T))
    plain = dict(w)
    del plain["pre_norm_w"]
    assert _rel(out, orc.moe_forward(x, ids, tw, plain).float()) > 0.05   # the norm is not a no-op here


@pytest.mark.parametrize("T,H,post,given,sigmoid", [
    (1, 1280, True, False, False),     # four warps norm one row: sums of squares across warps, an odd number of 256-column steps
    (1, 256, False, True, False),      # most lanes of those warps have nothing
    (2, 1280, False, False, True),     # two warps a row; sigmoid weights and selection bias
    (3, 768, True, False, True),       # a warp a row
    (4, 2304, True, True, False),
    (5, 1280, False, False, True),     # warps come round for a second row, the last round partly
    (6, 4096, True, True, False)])
def test_few_token_kernel_with_pre_expert_norm_and_sigmoid_routing(cuda_dev, T, H, post, given, sigmoid):
    """moe_few_kernel norms the token rows in its prologue in a form that depends on the token count; its top-k must give
    the ids and weights of the routing kernel, bit for bit, in both modes. Twice on one state."""
    m, inputs, _lib, orc = _mods()
    I, E, k = 512, 16, 4
    w = inputs.make_weights(H, I, E, 73, cuda_dev, post_norm=post)
    g = torch.Generator(device=cuda_dev).manual_seed(T + H)
    w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    if sigmoid:
        w["route_bias"] = torch.randn((E,), generator=g, device=cuda_dev) * 0.05
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=8, routing_mode="sigmoid_bias" if sigmoid else "softmax_topk")
    fits = ctypes.c_int(0)
    assert st["lib"].lib.msk_moe_few_fits(ctypes.byref(st["cfg"]), T, 2 + int(given), ctypes.byref(fits)) == 0 and fits.value == 1
    for _ in range(2):
        x = (torch.randn((T, H), generator=g, device=cuda_dev) * 3.0).to(torch.bfloat16)
        data = {"hidden_states": x, "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
        ids, tw = m._route(data, st, x, T)
        if given:
            out = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, st)
        else:
            out, got_ids, got_tw = m.kernel_fn(data, st, return_routing=True)
            assert torch.equal(got_ids, ids) and torch.equal(got_tw, tw)
        torch.cuda.synchronize()
        assert m.read_status(st) == 0
        rid, rtw = orc.route_topk(data["router_logits"].cpu(), k, "sigmoid_bias" if sigmoid else "softmax_topk",
                                  w["route_bias"].cpu() if sigmoid else None)
        assert torch.equal(ids.cpu(), rid) and torch.allclose(tw.cpu(), rtw, rtol=1e-5)    # expf and a sum of four: some 1e-6
        ref, parts = orc.moe_forward(x, ids, tw, w, return_parts=True)
        _check_forward(out, ref, parts, m.workspace_views(st, T))


@pytest.mark.parametrize("T,routed", [(2, False), (3, True)])
def test_few_token_kernel_shares_pinned_rows_of_several_tokens(cuda_dev, T, routed):
    """HostMappedStep at two and three tokens: several CTAs' slices make up a row, two warps or one copy it."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1280, 512, 16, 2
    st = m.prepare(inputs.make_weights(H, I, E, 74, cuda_dev, post_norm=routed), n_experts=E, top_k=k, max_tokens=8)
    fits = ctypes.c_int(0)
    assert st["lib"].lib.msk_moe_few_fits(ctypes.byref(st["cfg"]), T, 4 + int(routed), ctypes.byref(fits)) == 0 and fits.value == 1
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    datas = []
    for _ in range(6):
        d = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)}
        logits = torch.randn((T, E), generator=g, device=cuda_dev)
        if routed:
            tw, ids = torch.softmax(logits, dim=-1).topk(k, dim=-1)
            d["topk_ids"], d["topk_weights"] = ids.to(torch.int32), tw.contiguous()
        else:
            d["router_logits"] = logits
        datas.append(d)
    step = m.HostMappedStep(st, {key: v.cpu() for key, v in datas[0].items()})
    for d in datas:
        want = m.kernel_fn(d, st)
        got = step({key: v.cpu() for key, v in d.items()})
        step.done.synchronize()
        assert torch.equal(got, want.cpu())
    assert m.read_status(st) == 0


@pytest.mark.parametrize("T", [64, 8192])
def test_full_size_properties(cuda_dev, T):
    """Benchmark-size shapes (H4096 I1536 E128 top-8; T = 64 decode sweep point, T = 8192 prefill),
    where the CPU oracle would take minutes: properties that hold whatever the size.
    (1) A token's output does not depend on where the token sits: permuting the tokens permutes
    the output rows, bit for bit. (2) Halving the top-k weights halves the output exactly.
    (3) Tokens whose ids are all -1 come out zero and leave the other tokens' rows untouched."""
    m, inputs, _lib, orc = _mods()
    s = inputs.SHAPES["decode"]
    H, I, E, k = s["H"], s["I"], s["E"], s["k"]
    w = inputs.make_weights_random_bytes(H, I, E, 5, cuda_dev)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    data, _ = inputs.make_inputs("prefill" if T > 256 else "decode", T, 3, cuda_dev)
    x, logits = data["hidden_states"], data["router_logits"]
    out, ids, tw = m.kernel_fn({"hidden_states": x, "router_logits": logits}, st, return_routing=True)
    out = out.clone()
    g = torch.Generator(device=cuda_dev).manual_seed(1)
    p = torch.randperm(T, generator=g, device=cuda_dev)
    out_p = m.kernel_fn({"hidden_states": x[p].contiguous(), "router_logits": logits[p].contiguous()}, st)
    assert torch.equal(out_p, out[p])
    half = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw * 0.5}, st)
    assert torch.equal(half.float() * 2.0, out.float())
    ids2 = ids.clone()
    ids2[::7] = -1
    z = m.kernel_fn({"hidden_states": x, "topk_ids": ids2, "topk_weights": tw}, st)
    assert float(z[::7].float().abs().max()) == 0.0
    keep = torch.ones(T, dtype=torch.bool, device=cuda_dev)
    keep[::7] = False
    assert torch.equal(z[keep], out[keep])
    torch.cuda.synchronize()
    assert m.read_status(st) == 0


def _oracle_rows_of_tokens(orc, w, x, ids, tw, sel, post_norm=False):
    """Oracle evaluation of the tokens `sel` of a larger call: all of their experts (a dense local
    table over the touched ones). Returns (out bf16 [len(sel), H], parts, entry map): parts as
    orc.moe_forward returns them, and for every oracle row q' the (token index in sel, slot) it is."""
    sel_l = sel.tolist()
    sub_ids = ids[sel].cpu()
    touched = sorted(set(int(v) for v in sub_ids.flatten().tolist() if v >= 0))
    remap = {e: j for j, e in enumerate(touched)}
    lids = torch.tensor([[remap.get(int(v), -1) for v in row] for row in sub_ids.tolist()], dtype=torch.int32)

    def take(t):   # fp8 tensors are indexed through their bytes
        if t.dtype == torch.float8_e4m3fn:
            return t.view(torch.uint8)[touched].view(torch.float8_e4m3fn).cpu()
        return t[touched].cpu()

    sub = {key: take(w[key]) for key in ("w13", "w13_sf", "w13_gs", "w2", "w2_sf", "w2_gs")}
    if post_norm:
        sub["post_norm_w"] = w["post_norm_w"].cpu()
    ref, parts = orc.moe_forward(x[sel].cpu(), lids, tw[sel].cpu(), sub, return_parts=True)
    return ref, parts, sel_l


@pytest.mark.parametrize("T", [64, 8192])
def test_full_size_outputs_match_oracle_on_sampled_tokens(cuda_dev, T):
    """The benchmarked configurations themselves (H4096 I1536 E128 top-8; T = 64 with the 16-token
    tile, T = 8192 Zipf-routed with the 128-token tile and 16 K stages): eight tokens of the real
    output, and their rows of `inter` and `y` in the workspace, against the oracle evaluated on all
    of those tokens' experts."""
    m, inputs, _lib, orc = _mods()
    s = inputs.SHAPES["decode"]
    H, I, E, k = s["H"], s["I"], s["E"], s["k"]
    w = inputs.make_weights_random_bytes(H, I, E, 5, cuda_dev)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    data, _ = inputs.make_inputs("prefill" if T > 256 else "sweep", T, 3, cuda_dev)
    x, logits = data["hidden_states"], data["router_logits"]
    out, ids, tw = m.kernel_fn({"hidden_states": x, "router_logits": logits}, st, return_routing=True)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    views = m.workspace_views(st, T)
    rid, _ = orc.route_topk(logits.cpu(), k)
    assert torch.equal(ids.cpu(), rid)
    sel = torch.arange(0, T, max(T // 8, 1))[:8]
    ref, parts, _ = _oracle_rows_of_tokens(orc, w, x, ids, tw, sel)
    assert _rel(out[sel.to(cuda_dev)], parts["out_fp32"]) <= TOL
    inv = views["inv"].cpu().view(T, k)
    rows_gpu = []
    for q in range(int(parts["off"][-1])):
        entry = int(parts["perm"][q])
        rows_gpu.append(int(inv[int(sel[entry // k]), entry % k]))
    rows_gpu = torch.tensor(rows_gpu, device=views["y"].device)
    assert _rel(views["inter"][rows_gpu], parts["inter"]) <= TOL
    assert _rel(views["y"][rows_gpu], parts["y"]) <= TOL


@pytest.mark.parametrize("T,tile", [(64, 16), (600, 128), (200, 64)])
def test_forward_expert_parallel_shape(cuda_dev, T, tile):
    """The per-expert shape of the expert-parallel configuration (H7168 I2048: 28 K stages for the
    gate/up GEMM, 8 for the down GEMM, 28 pairs of down tiles), four local experts of eight, top-4,
    with the narrow and the wide token tile."""
    m, inputs, _lib, orc = _mods()
    out, ref, parts, views, st, _ = _run_forward(m, inputs, orc, cuda_dev, 7168, 2048, 8, 4, T, seed=300 + T,
                                                 post_norm=True, lo=2, nloc=4, token_tile=tile)
    assert m.plan(st, T)[0] == tile
    _check_forward(out, ref, parts, views)


@pytest.mark.parametrize("tile", [0, 64, 16])
def test_forward_reference_skewed_counts(cuda_dev, tile):
    """The reference's own expert check (muse_prefill_layer/py/07_selftest.py:41-73): T = 700, counts
    [300, 200, 100, 60, 33, 17, 14, 5, 1] over nine experts, entries laid out as its
    `_routes_from_counts` does (entry idx of expert e's c-th row: token idx % T, slot idx // T; all
    other slots -1)."""
    m, inputs, _lib, orc = _mods()
    H, I, k, T = 1024, 512, 8, 700
    counts = [300, 200, 100, 60, 33, 17, 14, 5, 1]
    E = len(counts)
    ids = torch.full((T * k,), -1, dtype=torch.int32)
    r = 0
    for e, c in enumerate(counts):
        idx = torch.arange(r, r + c)
        ids[(idx % T) * k + idx // T] = e
        r += c
    ids = ids.view(T, k).to(cuda_dev)
    w = inputs.make_weights(H, I, E, 91, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, token_tile=tile)
    g = torch.Generator(device=cuda_dev).manual_seed(17)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    tw = torch.rand((T, k), generator=g, device=cuda_dev)
    out = m.kernel_fn({"hidden_states": x, "topk_ids": ids, "topk_weights": tw}, st)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    ref, parts = orc.moe_forward(x, ids, tw, w, return_parts=True)
    assert parts["cnt"].tolist() == counts
    _check_forward(out, ref, parts, m.workspace_views(st, T))


SENTINEL = 0x5EADBEEF
GUARD_WORDS = 65536


def _guarded(t):
    """Copy of tensor t placed in front of 64 Ki sentinel words (the reference's guard scheme,
    muse_decode_layer/py/05_tune.py:453-477). Returns (view with t's shape and dtype, guard words)."""
    nbytes = t.numel() * t.element_size()
    pad = (nbytes + 255) // 256 * 256
    buf = torch.empty(pad + GUARD_WORDS * 4, dtype=torch.uint8, device=t.device)
    guard = buf[pad:].view(torch.int32)
    guard.fill_(SENTINEL)
    buf[nbytes:pad].view(torch.uint8).fill_(0xA5)
    view = buf[:nbytes].view(t.dtype).view(t.shape)
    view.copy_(t)
    return view, guard, buf[nbytes:pad]


@pytest.mark.parametrize("I,cap,sequence", [(512, 256, (32, 16, 256, 8, 16, 128, 16)),
                                            (1536, 700, (8, 700, 40, 2, 256, 48, 8, 130, 4, 40))])   # FP4, pair and few-token kernel, 64-token tile in turn
def test_state_hygiene_token_sequence_and_guard_words(cuda_dev, I, cap, sequence):
    """One state driven through the reference's token-count sequence 32, 16, 256, 8, 16, 128, 16
    (muse_decode_layer/py/17_moev.py:882-908): every output must equal, bit for bit, the output of a
    freshly prepared state on the same input (nothing a call leaves in the workspace may leak into the
    next), and 64 Ki sentinel words behind the output, the workspace and both packed weight buffers
    must survive every call."""
    m, inputs, _lib, orc = _mods()
    H, E, k = 1024, 16, 4
    w = inputs.make_weights(H, I, E, 123, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=cap)
    guards = []
    for key in ("workspace", "packed13", "packed2"):
        st[key], g, pad = _guarded(st[key])
        guards.append((key, g, pad))
    for step, T in enumerate(sequence):
        g = torch.Generator(device=cuda_dev).manual_seed(500 + step)
        data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
                "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
        out_buf, out_guard, out_pad = _guarded(torch.empty((T, H), dtype=torch.bfloat16, device=cuda_dev))
        got = m.kernel_fn(data, st, out=out_buf)
        fresh = m.prepare(w, n_experts=E, top_k=k, max_tokens=cap)
        want = m.kernel_fn(data, fresh)
        torch.cuda.synchronize()
        assert torch.equal(got, want), (step, T)
        assert m.read_status(st) == 0 and m.read_status(fresh) == 0
        for key, gw, pad in guards + [("out", out_guard, out_pad)]:
            assert bool((gw == SENTINEL).all()), (step, T, key)
            assert bool((pad == 0xA5).all()), (step, T, key)
        if step == 0:   # and the first one against the oracle, so "equal" is not "equally wrong"
            _, ids, tw = m.kernel_fn(data, fresh, return_routing=True)
            ref = orc.moe_forward(data["hidden_states"], ids, tw, w).float()
            assert _rel(got, ref) <= TOL


def test_bounded_wait_runs_out_cleanly_and_the_state_recovers(cuda_dev):
    """Failure detection without a fault: the streaming probe is told to withhold one slot release, so
    its producer's bounded wait (one second) runs out; the kernel must come back by itself with the
    time-out status, leave the context usable, and the library must work normally afterwards. Then the
    recovery path of a state: a workspace whose control words were left dirty (as a kernel that gave
    up would leave them) is put back by reinit_workspace and gives the clean result again."""
    import time

    m, inputs, _lib, orc = _mods()
    t0 = time.time()
    gbs, status = m.bw_probe(nbytes=64 << 20, skip_release=2, device=cuda_dev)
    assert status == 1                       # MSK_DEV_ERR_TIMEOUT, reported, not trapped
    assert 0.5 < time.time() - t0 < 30.0     # the one-second limit, not an endless spin
    gbs, status = m.bw_probe(nbytes=256 << 20, device=cuda_dev)
    assert status == 0 and gbs > 500.0       # the context is alive and the same kernel streams again
    H, I, E, k, T = 1024, 512, 16, 4, 8
    w = inputs.make_weights(H, I, E, 7, cuda_dev, post_norm=True)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=32, flat_shares=1, decode_path=1)
    g = torch.Generator(device=cuda_dev).manual_seed(3)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    clean = m.kernel_fn(data, st).clone()
    torch.cuda.synchronize()
    views = {}
    for which in (7, 8, 10):                 # unit tickets, control words of the few-token paths, tile hand-over counters
        ptr = ctypes.c_void_p()
        _lib.check(st["lib"].lib.msk_moe_workspace_view(ctypes.byref(st["cfg"]), _lib.ptr(st["workspace"]), which,
                                                        ctypes.byref(ptr)), "view")
        views[which] = ptr.value - st["workspace"].data_ptr()
    st["workspace"][views[7]:views[7] + 64].fill_(1)      # tickets half-way
    st["workspace"][views[8]:views[8] + 8192].fill_(3)    # token tickets, grid and tile counters
    st["workspace"][views[10]:views[10] + 64].fill_(5)    # gate/up units counted for tiles that no down unit took over
    st["workspace"][:4].copy_(torch.tensor([1, 0, 0, 0], dtype=torch.uint8))   # sticky status word
    assert m.read_status(st) == 1
    m.reinit_workspace(st)
    assert m.read_status(st) == 0
    for path in (1, 3):
        st["cfg"].decode_path = path
        got = m.kernel_fn(data, st)
        assert torch.equal(got, clean) if path == 1 else _rel(got, clean) <= 8e-3
        torch.cuda.synchronize()
        assert m.read_status(st) == 0


@pytest.mark.parametrize("T,post", [(1, False), (2, True)])
def test_few_token_kernel_gives_up_cleanly_and_recovers(cuda_dev, T, post):
    """A tile counter of the few-token kernel left one short (what a step that gave up can leave behind): the down units'
    wait for that tile runs out (one second), the kernel comes back by itself with the time-out status, the
    context stays usable, and after reinit_workspace the state gives the clean bits again."""
    m, inputs, _lib, orc = _mods()
    # every team has three gate/up units to do before its first down unit (with H = 1024 those of 64 CTAs have none, and ask at once)
    H, I, E, k = 4096, 4096, 16, 8
    w = inputs.make_weights(H, I, E, 8, cuda_dev, post_norm=post)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=8)
    g = torch.Generator(device=cuda_dev).manual_seed(4)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    clean = m.kernel_fn(data, st).clone()
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    ptr = ctypes.c_void_p()
    _lib.check(st["lib"].lib.msk_moe_workspace_view(ctypes.byref(st["cfg"]), _lib.ptr(st["workspace"]), 8, ctypes.byref(ptr)),
               "view")
    tile0 = ptr.value - st["workspace"].data_ptr() + 4352     # per-tile counters of the few-token paths
    # the second tile's: its units are dealt in the first rounds, and its count is asked for behind a complete first one, by when some of them
    # have been counted (-1 itself passes for complete)
    tile = tile0 + 4
    st["workspace"][tile:tile + 4].fill_(255)                 # -1: the tile's last unit will not complete it
    m.kernel_fn(data, st)
    torch.cuda.synchronize()
    assert m.read_status(st) == 1
    m.reinit_workspace(st)
    for _ in range(2):
        assert torch.equal(m.kernel_fn(data, st), clean)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0


@pytest.mark.parametrize("ctas,rows", [(2, 64), (2, 200), (6, 64)])
def test_pair_kernel_gives_up_cleanly_and_recovers(cuda_dev, ctas, rows):
    """The same for the pair kernel: the first token tile's counter one short. Each cluster has announced gate/up units of that
    tile before it asks for the count (a place of its unit list is used again behind the announcement), so the wait of
    the tile's down units cannot be met and runs out; whole warps give up together and the status says so."""
    m, inputs, _lib, orc = _mods()
    H, I, E = 512, 1024 * (ctas // 2), 2
    w = inputs.make_weights(H, I, E, 8, cuda_dev)
    st = m.prepare(w, n_experts=E, top_k=1, max_tokens=2 * rows, token_tile=128, num_ctas=ctas)
    g = torch.Generator(device=cuda_dev).manual_seed(4)
    data = {"hidden_states": torch.randn((2 * rows, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "topk_ids": torch.arange(2 * rows, device=cuda_dev, dtype=torch.int32).remainder(2).reshape(-1, 1).contiguous(),
            "topk_weights": torch.ones((2 * rows, 1), device=cuda_dev)}
    clean = m.kernel_fn(data, st).clone()
    assert m.read_status(st) == 0
    ptr = ctypes.c_void_p()
    _lib.check(st["lib"].lib.msk_moe_workspace_view(ctypes.byref(st["cfg"]), _lib.ptr(st["workspace"]), 10, ctypes.byref(ptr)), "view")
    tile0 = ptr.value - st["workspace"].data_ptr()
    st["workspace"][tile0:tile0 + 4].fill_(255)
    m.kernel_fn(data, st)
    assert m.read_status(st) == 1
    m.reinit_workspace(st)
    for _ in range(2):
        assert torch.equal(m.kernel_fn(data, st), clean)
    assert m.read_status(st) == 0


def test_state_dict_round_trip_skips_the_repack(cuda_dev):
    """state_dict() / load_state_dict(): the packed tiles, scales and configuration are enough to
    rebuild a state; kernel_fn on the rebuilt state gives the same bits."""
    import copy
    import io

    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 1024, 512, 8, 2, 40
    w = inputs.make_weights(H, I, E, 19, cuda_dev, post_norm=True)
    g = torch.Generator(device=cuda_dev).manual_seed(5)
    w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    w["router"] = torch.randn((E, H), generator=g, device=cuda_dev) * 0.02
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=64, routing_mode="softmax_topk")
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    want = m.kernel_fn({"hidden_states": x}, st)
    buf = io.BytesIO()
    torch.save(m.state_dict(st), buf)
    buf.seek(0)
    st2 = m.load_state_dict(torch.load(buf, map_location="cpu"), device=cuda_dev)
    assert st2["cfg"].hidden == H and st2["cfg"].max_tokens == 64
    assert torch.equal(m.kernel_fn({"hidden_states": x}, st2), want)
    assert torch.equal(m.kernel_fn({"hidden_states": x}, copy.deepcopy(st2)), want)
    back = m.export_weights(st2)
    assert torch.equal(back["w13"], w["w13"]) and torch.equal(back["w2_sf"], w["w2_sf"].view(torch.uint8))


def test_state_saved_with_the_host_inputs_field_loads(cuda_dev):
    """States saved while the configuration had a field host_inputs load like any other."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 512, 256, 8, 2, 3
    st = m.prepare(inputs.make_weights(H, I, E, 21, cuda_dev), n_experts=E, top_k=k, max_tokens=T)
    g = torch.Generator(device=cuda_dev).manual_seed(6)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    sd = m.state_dict(st)
    sd["config"] = dict(sd["config"], host_inputs=0)
    assert torch.equal(m.kernel_fn(data, m.load_state_dict(sd)), m.kernel_fn(data, st))


def test_state_saved_in_128_row_tiles_loads(cuda_dev):
    """A saved state without a layout number holds tiles of 128 rows x 256 K: loading puts them in the order the
    kernels read. The tiles are built here from the original weights."""
    m, inputs, _lib, orc = _mods()
    H, I, E = 768, 512, 3
    w = inputs.make_weights(H, I, E, 41, cuda_dev)
    st = m.prepare(w, n_experts=E, top_k=2, max_tokens=16)

    def tiles(codes, sf, first_rows):   # rows of each tile in the order of the tiles
        rows = torch.cat([torch.arange(r, r + 128) for r in first_rows]).to(cuda_dev)
        c = codes.view(torch.uint8)[:, rows].view(E, len(first_rows), 128, -1, 8, 16).permute(0, 1, 3, 4, 2, 5)
        s = sf.view(torch.uint8)[:, rows].view(E, len(first_rows), 128, -1, 1, 16).permute(0, 1, 3, 4, 2, 5)
        return torch.cat([c, s], dim=3).reshape(-1)

    sd = m.state_dict(st)
    assert sd.pop("packed_layout") == 2
    sd["packed13"] = tiles(w["w13"], w["w13_sf"], [g * I + j * 128 for j in range(I // 128) for g in (0, 1)])
    sd["packed2"] = tiles(w["w2"], w["w2_sf"], [j * 128 for j in range(H // 128)])
    st2 = m.load_state_dict(sd)
    assert torch.equal(st2["packed13"], st["packed13"]) and torch.equal(st2["packed2"], st["packed2"])
    sd["packed_layout"] = 3
    with pytest.raises(RuntimeError):
        m.load_state_dict(sd)


def test_prefill_moe_runs_the_prefill_layer_call_site(cuda_dev):
    """The prefill layer's expert step (muse_prefill_layer/py/04_moe_forward.py:6-52 followed by its
    combine): un-normed pooler rows, local ids with -1, routing weights in; pre-expert norm, both
    GEMMs, post-expert norm and weighted sum out. T = 700 with the reference's skewed counts."""
    m, inputs, _lib, orc = _mods()
    from muse_moe_w4a16.compat import PrefillMoe

    H, I, k, T = 1024, 512, 8, 700
    counts = [300, 200, 100, 60, 33, 17, 14, 5, 1]
    E = len(counts)
    lid = torch.full((T * k,), -1, dtype=torch.int32)
    pos = torch.zeros((T * k,), dtype=torch.int32)
    r = 0
    for e, c in enumerate(counts):
        idx = torch.arange(r, r + c)
        lid[(idx % T) * k + idx // T] = e
        pos[(idx % T) * k + idx // T] = torch.arange(c, dtype=torch.int32)
        r += c
    lid, pos = lid.view(T, k).to(cuda_dev), pos.view(T, k).to(cuda_dev)
    cnt = torch.tensor(counts, dtype=torch.int32, device=cuda_dev)
    w = inputs.make_weights(H, I, E, 23, cuda_dev, post_norm=True)
    g = torch.Generator(device=cuda_dev).manual_seed(29)
    w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    ext = PrefillMoe(m.prepare(w, local_start=0, n_experts=E, top_k=k, max_tokens=T))
    p = (torch.randn((T, H), generator=g, device=cuda_dev) * 2.0).to(torch.bfloat16)
    topw = torch.rand((T, k), generator=g, device=cuda_dev)
    moe_out = torch.full((T, H), float("nan"), dtype=torch.bfloat16, device=cuda_dev)
    ex = ext.moe_forward(p, lid, pos, cnt, T, topw, out=moe_out)
    ext.moe_combine(None, ex["rrow"], lid, topw, w["post_norm_w"], moe_out)
    torch.cuda.synchronize()
    ref, parts = orc.moe_forward(p, lid, topw, w, return_parts=True)
    assert _rel(moe_out, parts["out_fp32"]) <= TOL
    assert ex["out"].data_ptr() == moe_out.data_ptr()
    assert np.array_equal(ex["rrow"].tensor().cpu().numpy().reshape(-1), parts["inv"])


def _nvf4_takes(st, T):
    takes = ctypes.c_int(0)
    assert st["lib"].lib.msk_moe_nvf4_takes(ctypes.byref(st["cfg"]), T, int(st["post_norm_w"] is not None) + 2 * int(st["pre_norm_w"] is not None), ctypes.byref(takes)) == 0
    return takes.value == 1


def _ids_of_counts(counts, lo, k, dev):
    """Global ids [T, k] that give local expert e counts[e] rows (one local route a token, at any slot) and others dropped."""
    ids = torch.full((sum(counts), k), -1, dtype=torch.int32)
    rows = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts)).to(torch.int32) + lo
    g = torch.Generator().manual_seed(sum(counts))
    ids[torch.arange(len(rows)), torch.randint(0, k, (len(rows),), generator=g)] = rows[torch.randperm(len(rows), generator=g)]
    return ids.to(dev)


@pytest.mark.parametrize("H,I,counts,ctas,pre,post", [
    (256, 1536, [1, 8, 9, 16, 17, 24], 0, False, False),       # tiles of every width, one K stage: a unit shorter than any ring
    (768, 1536, [25, 0, 49, 5, 48, 1], 0, True, True),         # two and three tiles an expert, the last ones narrower
    (1024, 1536, [32, 33, 15, 48, 49, 64], 0, False, False),   # whole tiles, tiles with one row behind them
    (2304, 1792, [31, 24, 2, 0, 0, 7], 37, False, True),       # odd numbers of stages, fewer CTAs than rows
    (8192, 1536, [4, 0, 11, 0, 15, 0], 0, True, False),        # the longest rows, shared by several CTAs
    (6400, 2048, [40, 100, 9], 5, False, False),               # rows of more blocks than a CTA has threads; every ring wraps often
    (512, 4096, [28], 1, False, True),                         # one CTA waits for nobody but itself
    (768, 1536, [2, 0, 2], 0, False, True),                    # the fewest tokens it takes
    (2048, 1536, [130, 0, 160], 0, True, True),                # two rows a CTA: the second one is fetched while the first is split
])
def test_nvf4_kernel_at_tile_edges(cuda_dev, H, I, counts, ctas, pre, post):
    """moe_nvf4_kernel against the oracle where its tiles, rings and dealing can go wrong, twice on one state (bit for bit)."""
    m, inputs, _lib, orc = _mods()
    E, k, lo, n = 64, 2, 7, len(counts)
    w = inputs.make_weights(H, I, n, 61, cuda_dev, post_norm=post)
    g = torch.Generator(device=cuda_dev).manual_seed(H + I)
    if pre:
        w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    T = sum(counts)
    st = m.prepare(w, local_start=lo, n_experts=E, top_k=k, max_tokens=T, num_ctas=ctas)
    assert _nvf4_takes(st, T)
    x = (torch.randn((T, H), generator=g, device=cuda_dev) * 2.0).to(torch.bfloat16)
    d = {"hidden_states": x, "topk_ids": _ids_of_counts(counts, lo, k, cuda_dev),
         "topk_weights": torch.rand((T, k), generator=g, device=cuda_dev) + 0.1}
    out = m.kernel_fn(d, st).clone()
    views = m.workspace_views(st, T)
    again = m.kernel_fn(d, st)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0 and torch.equal(again, out)
    ref, parts = orc.moe_forward(x, d["topk_ids"], d["topk_weights"], w, local_start=lo, return_parts=True)
    assert parts["cnt"].tolist() == counts
    _check_forward(out, ref, parts, views)


@pytest.mark.parametrize("scale", [1.0, 3.0e-3])
def test_nvf4_kernel_is_no_further_from_64_bits_than_the_f16_kernel(cuda_dev, scale):
    """Both GEMMs on their own: inter against 64 bits from the same token rows (its rounding to BF16, 1.6e-3 and 2.8e-3, hides all
    else), y against 64 bits from each kernel's own inter: the digits hold every element, FP32 sums of a digit each lose less than those of the
    F16 kernel."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 4096, 1536, 8, 2, 48
    w = inputs.make_weights(H, I, E, 17, cuda_dev)
    g = torch.Generator(device=cuda_dev).manual_seed(5)
    x = (torch.randn((T, H), generator=g, device=cuda_dev) * scale).to(torch.bfloat16)
    d = {"hidden_states": x, "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    err = {}
    for tile in (0, 16):
        st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, token_tile=tile)
        assert _nvf4_takes(st, T) == (tile == 0)
        m.kernel_fn(d, st)
        torch.cuda.synchronize()
        v = m.workspace_views(st, T)
        dq13, dq2 = m.dequant_packed(st)
        off, perm = v["off"].tolist(), v["perm"].long() // k
        i64, y64 = torch.empty((T * k, I), dtype=torch.float64, device=cuda_dev), torch.empty((T * k, H), dtype=torch.float64, device=cuda_dev)
        for e in range(E):
            r = slice(off[e], off[e + 1])
            gu = x[perm[r]].double() @ dq13[e].double().T * w["w13_gs"][e].double()
            i64[r] = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
            y64[r] = v["inter"][r].double() @ dq2[e].double().T * w["w2_gs"][e].double()
        err[tile] = [float((a.double() - b).norm() / b.norm()) for a, b in ((v["inter"], i64), (v["y"], y64))]
    assert err[0][0] <= err[16][0] * 1.001 and err[0][0] <= 4.0e-3, err
    assert err[0][1] <= err[16][1] and err[0][1] <= 2.0e-6, err
    print(err)


def test_nvf4_kernel_without_a_local_route(cuda_dev):
    """A rank's step none of whose tokens go to its experts: zeros, a clean status and a state whose next step gives the clean bits."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, lo, n, T = 768, 1536, 64, 2, 7, 3, 40
    w = inputs.make_weights(H, I, n, 33, cuda_dev)
    st = m.prepare(w, local_start=lo, n_experts=E, top_k=k, max_tokens=T)
    assert _nvf4_takes(st, T)
    g = torch.Generator(device=cuda_dev).manual_seed(2)
    d = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
         "topk_ids": _ids_of_counts([20, 0, 20], lo, k, cuda_dev), "topk_weights": torch.rand((T, k), generator=g, device=cuda_dev)}
    clean = m.kernel_fn(d, st).clone()
    away = torch.full((T, k), -1, dtype=torch.int32, device=cuda_dev)
    away[::2] = lo + n
    none = m.kernel_fn(dict(d, topk_ids=away), st)
    assert not bool(none.any()) and torch.equal(m.kernel_fn(d, st), clean)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0


@pytest.mark.parametrize("T,pre", [(8, False), (8, True), (40, False)])
def test_nvf4_kernel_replayed_behind_the_kernel_that_writes_its_rows(cuda_dev, T, pre):
    """Its CTAs read their first token row in front of their wait for the sort: rows that the launch before the step writes, other ones with
    every replay and replay behind replay, against steps on their own; and the same rows in pinned host memory."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 1536, 16, 4
    w = inputs.make_weights(H, I, E, 71, cuda_dev, post_norm=True)
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    if pre:
        w["pre_norm_w"] = (torch.randn((H,), generator=g, device=cuda_dev) * 0.1).to(torch.bfloat16)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    assert _nvf4_takes(st, T)
    rows = torch.randn((8, T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    logits = torch.randn((8, T, E), generator=g, device=cuda_dev)
    a, b, x, l = rows[0].clone(), logits[0].clone(), torch.empty_like(rows[0]), torch.empty_like(logits[0])
    m.kernel_fn({"hidden_states": a, "router_logits": b}, st)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        torch.mul(b, 1.0, out=l)
        torch.mul(a, 1.0, out=x)
        out = m.kernel_fn({"hidden_states": x, "router_logits": l}, st)
    got = []
    for r, s in zip(rows, logits):
        a.copy_(r)
        b.copy_(s)
        graph.replay()
        got.append(out.clone())
    for r, s, y in zip(rows, logits, got):
        want, ids, tw = m.kernel_fn({"hidden_states": r, "router_logits": s}, st, return_routing=True)
        assert torch.equal(y, want)
        host = r.cpu().pin_memory()
        m._forward(st, st["cfg"], st["lib"].lib, host.data_ptr(), None, ids.data_ptr(), tw.data_ptr(), out.data_ptr(), T)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert m.read_status(st) == 0


def _wide_rows(T, H, g, dev):
    """Token rows with BF16 values from 2^-24 to the end of the F16 range side by side, three kinds in turn: any magnitudes, one
    magnitude in every block of sixteen far above the others (the largest on either side of a power of two), normal values."""
    mant = 1.0 + torch.randint(0, 128, (T, H), generator=g, device=dev) / 128.0
    x = mant * torch.exp2(torch.randint(-24, 16, (T, H), generator=g, device=dev).float())
    top = torch.tensor([1.0, 1.6953125, 1.703125, 1.7109375, 1.9921875], device=dev)[torch.randint(0, 5, (T, H // 16), generator=g, device=dev)]
    top = top * torch.exp2(torch.randint(-6, 16, (T, H // 16), generator=g, device=dev).float())
    low = top[:, :, None] * torch.exp2(-torch.randint(9, 26, (T, H // 16, 16), generator=g, device=dev).float()) * mant.view(T, H // 16, 16)
    low[:, :, 5] = top
    x[1::3] = low.view(T, H)[1::3]
    x[2::3] = torch.randn((T, H), generator=g, device=dev)[2::3].abs()
    return (x * (torch.randint(0, 2, (T, H), generator=g, device=dev) * 2 - 1)).to(torch.bfloat16)


@pytest.mark.parametrize("tile", [0, 16])
def test_activations_enter_the_gemms_exactly(cuda_dev, tile):
    """Experts that hand their row through: gate x[0] = 32, up x[i] / 32, so inter = x, and y = inter. Whatever lies beside an element
    in its row, what comes out is its F16 value, bit for bit, by the FP4 kernel as by the F16 one."""
    m, inputs, _lib, orc = _mods()
    H, E, k, T = 1536, 8, 1, 90
    eye = torch.zeros((H, H), dtype=torch.uint8, device=cuda_dev)
    eye.fill_diagonal_(2)                                         # E2M1 code of 1
    gate = torch.zeros_like(eye)
    gate[:, 0] = 2
    pack = lambda c: (c[:, 0::2] | (c[:, 1::2] << 4)).expand(E, -1, -1).contiguous()  # noqa: E731
    sf13 = torch.full((E, 2 * H, H // 16), 0x38, dtype=torch.uint8, device=cuda_dev)      # 1
    sf13[:, H:] = 0x10                                            # 2^-5
    one = torch.ones(E, device=cuda_dev)
    w = {"w13": pack(torch.cat([gate, eye])), "w13_sf": sf13, "w13_gs": one, "w2": pack(eye),
         "w2_sf": torch.full((E, H, H // 16), 0x38, dtype=torch.uint8, device=cuda_dev), "w2_gs": one}
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, token_tile=tile)
    assert _nvf4_takes(st, T) == (tile == 0)
    g = torch.Generator(device=cuda_dev).manual_seed(31)
    x = _wide_rows(T, H, g, cuda_dev)
    x[:, 0] = 32.0
    d = {"hidden_states": x, "topk_ids": _ids_of_counts([24, 1, 0, 33, 8, 17, 0, 7], 0, k, cuda_dev),
         "topk_weights": torch.ones((T, k), device=cuda_dev)}
    for _ in range(2):
        m.kernel_fn(d, st)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    v = m.workspace_views(st, T)
    want = x.half()[v["perm"].long()]
    assert torch.equal(v["inter"], want)
    assert torch.equal(v["y"], want.float())


@pytest.mark.parametrize("counts", [[1, 2, 3, 4, 5, 8, 9, 12], [4, 4, 4, 4, 4, 4, 4, 3], [17, 18, 19, 20, 4, 3, 2, 1]])
def test_nvf4_tiles_with_room_for_four_rows_hold_every_level(cuda_dev, counts):
    """Tiles of one to four rows, alone and behind whole ones, beside wider tiles: experts that hand their row through (gate x[0] = 32, up x[i] / 32),
    rows with second and third levels of digits in every K stage; y and inter bit for bit, twice."""
    m, inputs, _lib, orc = _mods()
    H, E, k, T = 1536, 8, 1, sum(counts)
    eye = torch.zeros((H, H), dtype=torch.uint8, device=cuda_dev)
    eye.fill_diagonal_(2)                                         # E2M1 code of 1
    gate = torch.zeros_like(eye)
    gate[:, 0] = 2
    pack = lambda c: (c[:, 0::2] | (c[:, 1::2] << 4)).expand(E, -1, -1).contiguous()  # noqa: E731
    sf13 = torch.full((E, 2 * H, H // 16), 0x38, dtype=torch.uint8, device=cuda_dev)      # 1
    sf13[:, H:] = 0x10                                            # 2^-5
    one = torch.ones(E, device=cuda_dev)
    w = {"w13": pack(torch.cat([gate, eye])), "w13_sf": sf13, "w13_gs": one, "w2": pack(eye),
         "w2_sf": torch.full((E, H, H // 16), 0x38, dtype=torch.uint8, device=cuda_dev), "w2_gs": one}
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    assert _nvf4_takes(st, T)
    g = torch.Generator(device=cuda_dev).manual_seed(37)
    x = _wide_rows(T, H, g, cuda_dev)
    x[:, 0] = 32.0
    d = {"hidden_states": x, "topk_ids": _ids_of_counts(counts, 0, k, cuda_dev), "topk_weights": torch.ones((T, k), device=cuda_dev)}
    for _ in range(2):
        m.kernel_fn(d, st)
        torch.cuda.synchronize()
        assert m.read_status(st) == 0
        v = m.workspace_views(st, T)
        want = x.half()[v["perm"].long()]
        assert torch.equal(v["inter"], want)
        assert torch.equal(v["y"], want.float())


@pytest.mark.parametrize("large", [1000.0, 20000.0])
def test_nvf4_kernel_beside_large_channels_that_the_weights_ignore(cuda_dev, large):
    """Every sixteenth channel large, in the token rows and in inter, the others orders below, and weights of zero
    for the large ones: sums against 64 bits, no further off than the F16 kernel's."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 4096, 1536, 8, 2, 48
    w = inputs.make_weights(H, I, E, 17, cuda_dev)
    w["w13"].view(torch.uint8)[:, :, 2::8] &= 0xF0                # codes of channels 4, 20, 36 ...
    w["w2"].view(torch.uint8)[:, :, 2::8] &= 0xF0
    sf = w["w13_sf"].view(torch.uint8)
    small = torch.arange(I, device=cuda_dev) % 16 != 4            # gate and up rows of the other channels: 2^-4
    sf[:, small.repeat(2)] = (sf[:, small.repeat(2)].int() - 0x20).clamp(min=1).to(torch.uint8)
    w["w13_gs"] *= 16.0
    g = torch.Generator(device=cuda_dev).manual_seed(5)
    x = torch.randn((T, H), generator=g, device=cuda_dev)
    x[:, 4::16] *= large
    d = {"hidden_states": x.to(torch.bfloat16), "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    x = d["hidden_states"].float().clamp(-65504.0, 65504.0).half().double()
    err, spread = {}, 0.0
    for tile in (0, 16):
        st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, token_tile=tile)
        assert _nvf4_takes(st, T) == (tile == 0)
        m.kernel_fn(d, st)
        torch.cuda.synchronize()
        v = m.workspace_views(st, T)
        dq13, dq2 = m.dequant_packed(st)
        off, perm = v["off"].tolist(), v["perm"].long() // k
        i64, y64 = torch.empty((T * k, I), dtype=torch.float64, device=cuda_dev), torch.empty((T * k, H), dtype=torch.float64, device=cuda_dev)
        for e in range(E):
            r = slice(off[e], off[e + 1])
            gu = x[perm[r]] @ dq13[e].double().T * w["w13_gs"][e].double()
            i64[r] = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
            y64[r] = v["inter"][r].double() @ dq2[e].double().T * w["w2_gs"][e].double()
        spread = float(v["inter"][:, ~small].double().norm() / v["inter"][:, small].double().norm())
        err[tile] = [float((a.double() - b).norm() / b.norm()) for a, b in ((v["inter"][:, small], i64[:, small]), (v["y"], y64))]
    assert spread > 50.0, (spread, err)
    assert err[0][0] <= err[16][0] * 1.001 and err[0][0] <= 4.0e-3, err
    assert err[0][1] <= err[16][1] and err[0][1] <= 2.0e-6, err


def test_nvf4_kernel_with_negative_and_nan_scales_and_tokens_out_of_range(cuda_dev):
    """What the FP4 operands cannot hold as such: scale bytes with the sign bit (the codes take the sign), NaN scales, and tokens
    with NaN, infinite and huge elements, a zero row and values far below the row's largest. The F16 kernel is the reference: the
    same NaN places, close elsewhere."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 768, 1536, 8, 2, 40
    w = inputs.make_weights(H, I, E, 23, cuda_dev)
    g = torch.Generator(device=cuda_dev).manual_seed(9)
    for key in ("w13_sf", "w2_sf"):
        b = w[key].view(torch.uint8)
        b |= (torch.rand(b.shape, generator=g, device=cuda_dev) < 0.3).to(torch.uint8) << 7
    w["w2_sf"].view(torch.uint8)[3, 5, 7] = 0x7F
    w["w2_sf"].view(torch.uint8)[6, 700, 0] = 0xFF
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    x[1] = 0.0
    x[2, 3] = float("nan")
    x[3, 100] = float("inf")
    x[4, 50:60] = -3.0e38
    x[5, 1:] *= 1.0e-6
    d = {"hidden_states": x, "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    got = {}
    for tile in (0, 16):
        st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T, token_tile=tile)
        assert _nvf4_takes(st, T) == (tile == 0)
        out = m.kernel_fn(d, st).float()
        torch.cuda.synchronize()
        assert m.read_status(st) == 0
        got[tile] = (out, m.workspace_views(st, T)["y"])
    for a, b in zip(got[0], got[16]):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and bool(torch.isnan(a).any())
    (a, ya), (b, yb) = got[0], got[16]
    row = lambda v: v.nan_to_num(0.0).norm(dim=1)  # noqa: E731
    assert bool((row(a - b) <= TOL * row(b)).all())
    assert float(a[1].nan_to_num(0.0).abs().max()) == 0.0


def test_nvf4_kernel_gives_up_cleanly_and_recovers(cuda_dev):
    """A unit counter that starts far behind the last unit: every CTA computes its first unit and finds no more, the warps that
    wait for whole tiles run into their limit of a second, the kernel reports it and returns, and after
    reinit_workspace the state gives the clean bits again."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 512, 1536, 16, 4, 24
    w = inputs.make_weights(H, I, E, 29, cuda_dev)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    assert _nvf4_takes(st, T)
    g = torch.Generator(device=cuda_dev).manual_seed(3)
    data = {"hidden_states": torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16),
            "router_logits": torch.randn((T, E), generator=g, device=cuda_dev)}
    clean = m.kernel_fn(data, st).clone()
    torch.cuda.synchronize()
    assert m.read_status(st) == 0
    ptr = ctypes.c_void_p()
    _lib.check(st["lib"].lib.msk_moe_workspace_view(ctypes.byref(st["cfg"]), _lib.ptr(st["workspace"]), 8, ctypes.byref(ptr)), "view")
    at = ptr.value - st["workspace"].data_ptr() + 4096        # units drawn
    st["workspace"][at:at + 4].copy_(torch.tensor([0, 0, 16, 0], dtype=torch.uint8))
    m.kernel_fn(data, st)
    torch.cuda.synchronize()
    assert m.read_status(st) == 1
    m.reinit_workspace(st)
    for _ in range(2):
        assert torch.equal(m.kernel_fn(data, st), clean)
    torch.cuda.synchronize()
    assert m.read_status(st) == 0


def test_activations_outside_the_f16_range_saturate_as_documented(cuda_dev):
    """The MMA operands are F16: a BF16 activation beyond +-65504 enters the GEMM as +-65504 (and one
    below 2^-24 as zero), and so does a SwiGLU value that large. The result must equal the oracle
    evaluated with its operands saturated the same way, and rows inside the range must not be affected
    by a saturating neighbour."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k, T = 512, 256, 8, 2, 6
    w = inputs.make_weights(H, I, E, 31, cuda_dev)
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=T)
    g = torch.Generator(device=cuda_dev).manual_seed(37)
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    x[1, 5] = 3.0e5          # beyond the F16 range
    x[1, 9] = -1.0e6
    x[2, 7] = 1.0e-9         # below the smallest F16 subnormal
    logits = torch.randn((T, E), generator=g, device=cuda_dev)
    out, ids, tw = m.kernel_fn({"hidden_states": x, "router_logits": logits}, st, return_routing=True)
    torch.cuda.synchronize()
    ref = orc.moe_forward(x, ids, tw, w, f16_operands=True).float()   # x and inter saturated as the F16 operands are
    assert torch.isfinite(out.float()).all()
    assert _rel(out, ref) <= TOL
    plain = orc.moe_forward(x, ids, tw, w).float()
    keep = [0, 2, 3, 4, 5]
    assert _rel(out[keep], plain[keep]) <= TOL


@pytest.mark.parametrize("T,E,H", [(16, 128, 512), (50, 256, 1024), (300, 8, 512), (1000, 128, 4096), (130, 384, 2048)])
def test_router_logits_gemm_on_the_hi_lo_pair(cuda_dev, T, E, H):
    """msk_moe_router_logits_hilo: the FP32 router weight as the reference's exact-sum BF16 pair
    (muse_decode_layer/py/05_tune.py:279-286) through the tensor-core GEMM. The logits must equal the
    FP64 product of x with hi + lo up to FP32 accumulation, stay within what w - hi - lo drops of the
    FP32 product, repeat bit for bit, and give the FP32 matvec's top-k except where two scores are
    closer than that difference (reported as tie-risk, not as a failure)."""
    m, inputs, _lib, orc = _mods()
    lib = _lib.load()
    g = torch.Generator(device=cuda_dev).manual_seed(T + E)
    w = torch.randn((E, H), generator=g, device=cuda_dev) * 0.02
    x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
    hilo = m.split_router(w)
    assert hilo.dtype == torch.bfloat16 and tuple(hilo.shape) == (2 * E, H)
    k = min(8, E)
    cfg = _lib.MskMoeCfg(hidden=H, inter=256, n_experts=E, local_start=0, local_count=min(E, 256), top_k=k, max_tokens=T)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_dev)

    def gemm():
        out = torch.full((T, E), float("nan"), device=cuda_dev)
        _lib.check(lib.msk_moe_router_logits_hilo(ctypes.byref(cfg), _lib.ptr(x), _lib.ptr(hilo), _lib.ptr(out),
                                                  _lib.ptr(status), T, st), "router_logits_hilo")
        return out

    a = gemm()
    b = gemm()
    mv = torch.empty((T, E), device=cuda_dev)
    _lib.check(lib.msk_moe_router_logits(ctypes.byref(cfg), _lib.ptr(x), _lib.ptr(w), _lib.ptr(mv), T, st), "router_logits")
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and torch.equal(a, b) and torch.isfinite(a).all()
    xd = x.double()
    pair = xd @ (hilo[:E].double() + hilo[E:].double()).T
    full = xd @ w.double().T
    scale = float(full.abs().max())
    assert float((a.double() - pair).abs().max()) <= 2e-5 * scale      # FP32 accumulation of exact products (up to 8192 of them)
    assert float((a.double() - full).abs().max()) <= 5e-5 * scale      # plus the part of w the pair drops
    ia, _ = orc.route_topk(a.cpu(), k)
    ib, _ = orc.route_topk(mv.cpu(), k)
    rows, slots = np.nonzero(ia.numpy() != ib.numpy())
    fl = full.cpu().numpy()
    for r, c in zip(rows, slots):      # tie-risk: the two candidates' exact scores are closer than the logits' error
        assert abs(fl[r, ia[r, c]] - fl[r, ib[r, c]]) <= 1e-4 * scale, (r, c)
    assert len(set(rows.tolist())) <= max(1, T // 50)


@pytest.mark.parametrize("T,E,H,off", [(5, 130, 768, 0), (15, 8, 256, 1), (263, 16, 4352, 0)])
def test_router_matvec_of_many_tokens_gives_the_bits_of_each_alone(cuda_dev, T, E, H, off):
    """msk_moe_router_logits: tokens are spread over blocks of four, the last one ragged; a token's logits are those of a
    call with that token alone, from aligned and (off = 1) element-aligned rows, and the FP64 product up to FP32 sums."""
    m, inputs, _lib, orc = _mods()
    lib = _lib.load()
    g = torch.Generator(device=cuda_dev).manual_seed(T)
    w = torch.randn((E, H), generator=g, device=cuda_dev) * 0.02
    x = torch.randn((T * H + off,), generator=g, device=cuda_dev).to(torch.bfloat16)[off:].view(T, H)
    cfg = _lib.MskMoeCfg(hidden=H, inter=256, n_experts=E, local_start=0, local_count=E, top_k=1, max_tokens=T)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def logits(rows):
        out = torch.full((rows.shape[0], E), float("nan"), device=cuda_dev)
        _lib.check(lib.msk_moe_router_logits(ctypes.byref(cfg), _lib.ptr(rows), _lib.ptr(w), _lib.ptr(out), rows.shape[0], st),
                   "router_logits")
        return out

    got = logits(x)
    for t in sorted({0, 3, 4, T // 2, T - 1}):
        assert torch.equal(got[t], logits(x[t:t + 1])[0])
    want = x.double() @ w.double().T
    # at most 32 products added up by a thread, five shuffle steps, eight warps: 45 roundings on the way of a product
    assert bool(((got.double() - want).abs() <= 45 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)).all())


@pytest.mark.parametrize("T,E,H", [(64, 130, 256),      # four K steps: four CTAs of one step; two tiles of experts
                                   (65, 8, 768),        # twelve steps over eight CTAs
                                   (2051, 128, 256)])   # 128-token tiles, the last with three tokens
def test_router_logits_split_over_a_cluster(cuda_dev, T, E, H):
    test_router_logits_gemm_on_the_hi_lo_pair(cuda_dev, T, E, H)


def test_kernel_fn_with_router_weight_uses_the_gemm_from_sixteen_tokens(cuda_dev):
    """weights["router"]: few tokens take the FP32 matvec, 16 and more the hi + lo GEMM; both feed the
    same routing and expert kernels, and the output matches the oracle on the routing the module used."""
    m, inputs, _lib, orc = _mods()
    H, I, E, k = 1024, 512, 16, 4
    w = inputs.make_weights(H, I, E, 41, cuda_dev)
    g = torch.Generator(device=cuda_dev).manual_seed(43)
    w["router"] = torch.randn((E, H), generator=g, device=cuda_dev) * 0.02
    st = m.prepare(w, n_experts=E, top_k=k, max_tokens=256)
    for T in (5, 16, 200):
        x = torch.randn((T, H), generator=g, device=cuda_dev).to(torch.bfloat16)
        out, ids, tw = m.kernel_fn({"hidden_states": x}, st, return_routing=True)
        torch.cuda.synchronize()
        assert m.read_status(st) == 0
        rid, _ = orc.route_topk(orc.router_logits(x.cpu(), w["router"].cpu()), k)
        assert float((ids.cpu() == rid).all(dim=1).float().mean()) >= 0.97      # near-ties may pick the neighbour
        ref = orc.moe_forward(x, ids, tw, w).float()
        assert _rel(out, ref) <= TOL
