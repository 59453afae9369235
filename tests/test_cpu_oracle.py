"""CPU tests: the oracle against the reference-generated golden vectors and hand-computed
known answers, the quantiser, and the host side of the C ABI (no GPU, no compute calls)."""
import ctypes
import os
import re

import numpy as np
import pytest
import torch

from oracle import moe_oracle as orc

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
GOLD = np.load(os.path.join(HERE, "golden", "reference_vectors.npz"))


# ------------------------------------------------------------ golden vectors
def test_nibble_order_matches_reference_split_nibbles():
    codes, rows = GOLD["nib_codes"], GOLD["nib_rows"]
    assert np.array_equal(orc.split_nibbles(codes[rows]), GOLD["nib_out"])


def test_e4m3_table_matches_reference_lut():
    lut = GOLD["e4m3_lut"].astype(np.int64) & 0xFFFF           # bf16 bits of value * 2^64
    vals = orc.e4m3_value(np.arange(256, dtype=np.uint8))
    want = torch.from_numpy(lut.astype(np.int16)).view(torch.bfloat16).float().numpy()
    nan = np.isnan(vals)
    assert list(np.nonzero(nan)[0]) == [0x7F, 0xFF]
    assert np.array_equal(np.isnan(want), nan)
    assert np.array_equal(vals[~nan].astype(np.float64) * 2.0 ** 64, want[~nan].astype(np.float64))


@pytest.mark.parametrize("bs", [4, 33])
def test_sort_on_reference_generated_routing(bs):
    ids = GOLD[f"gen{bs}_ids"]
    w = GOLD[f"gen{bs}_w"]
    assert ids.shape == (bs, 8) and np.allclose(w.sum(-1), 1.0, atol=1e-5)
    cnt, off, perm, inv = orc.sort_routes(ids, 0, 32)  # the reference rank owns experts 0..31
    flat = ids.reshape(-1)
    local = (flat >= 0) & (flat < 32)
    assert cnt.sum() == local.sum() == off[-1]
    # same answer as a stable sort of the local ids (the bit-exactness target of the kernel)
    lid = torch.from_numpy(np.where(local, flat, 1 << 20))
    order = torch.sort(lid, stable=True).indices.numpy()[: int(off[-1])]
    assert np.array_equal(perm, order)
    assert np.array_equal(inv[perm], np.arange(len(perm)))
    assert np.all(inv[~local] == -1)
    for e in range(32):
        seg = perm[off[e]:off[e + 1]]
        assert np.all(flat[seg] == e) and np.all(np.diff(seg) > 0)


# --------------------------------------------------------- known-answer tests
def test_e2m1_codes_known_answers():
    want = [0, .5, 1, 1.5, 2, 3, 4, 6, -0.0, -.5, -1, -1.5, -2, -3, -4, -6]
    got = orc.e2m1_value(np.arange(16, dtype=np.uint8))
    assert np.array_equal(got, np.array(want, dtype=np.float32))
    assert np.signbit(got[8])


@pytest.mark.parametrize("byte,value", [(0x00, 0.0), (0x01, 2.0 ** -9), (0x07, 7 * 2.0 ** -9), (0x08, 2.0 ** -6),
                                        (0x38, 1.0), (0x40, 2.0), (0x7E, 448.0), (0xB8, -1.0)])
def test_e4m3_known_answers(byte, value):
    assert float(orc.e4m3_value(np.uint8(byte))) == value


def test_dequant_known_answers_all_codes_times_scales():
    scales = [0x00, 0x01, 0x07, 0x08, 0x38, 0x40, 0x7E]
    sv = [0.0, 2.0 ** -9, 7 * 2.0 ** -9, 2.0 ** -6, 1.0, 2.0, 448.0]
    e2 = [0, .5, 1, 1.5, 2, 3, 4, 6]
    codes = np.array([[(2 * j) | ((2 * j + 1) << 4) for j in range(8)]] * len(scales), dtype=np.uint8)  # k = 0..15
    sf = np.array([[s] for s in scales], dtype=np.uint8)
    for gs in (1.0, 3.0e-5):
        got = orc.dequant(codes, sf, gs)
        for r, s in enumerate(sv):
            for k in range(16):
                want = np.float32((-1 if k >= 8 else 1) * e2[k % 8] * s) * np.float32(gs)
                assert got[r, k] == want


def test_quantiser_round_trip_and_tie_rule():
    from muse_moe_w4a16 import quant

    ties = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, -0.25, -5.0, 7.0, 0.0])
    codes = quant.e2m1_codes(ties)
    assert codes.tolist() == [0, 2, 2, 4, 4, 6, 6, 8, 14, 7, 0]  # ties go to the even code
    g = torch.Generator().manual_seed(0)
    w = (torch.randn((64, 256), generator=g) * 0.02).to(torch.bfloat16)
    c, s, gs = quant.quantize_nvfp4(w)
    assert c.shape == (64, 128) and s.shape == (64, 16)
    assert abs(float(gs) - float(w.float().abs().max()) / (6 * 448)) < 1e-12
    dq = orc.dequant(c.numpy(), s.numpy(), float(gs))
    blk = w.float().view(64, 16, 16).abs().amax(-1).numpy().repeat(16, -1).reshape(64, 256)
    assert np.all(np.abs(dq - w.float().numpy()) <= 0.26 * blk + 1e-12)  # half an E2M1 step at the block top
    assert 0x08 <= int(s.min()) and int(s.max()) <= 0x7E                  # normal scale bytes only (neither zero, subnormal nor NaN)


def test_route_topk_tie_rule_and_weights():
    logits = torch.tensor([[1.0, 3.0, 3.0, -1.0, 3.0, 0.5]])
    ids, w = orc.route_topk(logits, 3)
    assert ids.tolist() == [[1, 2, 4]]
    assert torch.allclose(w, torch.full((1, 3), 1 / 3))
    ids, w = orc.route_topk(logits, 2, "sigmoid_bias", bias=torch.tensor([0, 0, 0, 5.0, 0, 0]), scale=1.0)
    assert ids.tolist() == [[3, 1]]
    s = torch.sigmoid(torch.tensor([-1.0, 3.0]))
    assert torch.allclose(w[0], s / s.sum())


def test_moe_forward_against_dense_evaluation():
    """The grouped oracle equals a dense per-token evaluation of the same formula."""
    from muse_moe_w4a16 import inputs

    H, I, E, k, T = 256, 256, 4, 2, 6
    w = inputs.make_weights(H, I, E, 1, "cpu", post_norm=True)
    g = torch.Generator().manual_seed(2)
    x = torch.randn((T, H), generator=g).to(torch.bfloat16)
    ids, tw = orc.route_topk(torch.randn((T, E), generator=g), k)
    out, parts = orc.moe_forward(x, ids, tw, w, return_parts=True)
    ref = torch.zeros((T, H))
    for t in range(T):
        for s in range(k):
            e = int(ids[t, s])
            y = orc.expert_forward(x[t:t + 1], w["w13"][e], w["w13_sf"][e], w["w13_gs"][e], w["w2"][e], w["w2_sf"][e],
                                   w["w2_gs"][e])[0]
            y = y * (1 + w["post_norm_w"].float())
            y = y * torch.rsqrt(y.pow(2).mean() + 1e-8)
            ref[t] += tw[t, s] * y
    assert torch.allclose(parts["out_fp32"], ref, rtol=1e-5, atol=1e-6)
    # local-range filter: the two halves of the experts sum to the whole (partial sums, EP "filter" mode)
    lo = {key: (v[:2] if key != "post_norm_w" else v) for key, v in w.items()}
    hi = {key: (v[2:] if key != "post_norm_w" else v) for key, v in w.items()}
    _, p0 = orc.moe_forward(x, ids, tw, lo, local_start=0, return_parts=True)
    _, p1 = orc.moe_forward(x, ids, tw, hi, local_start=2, return_parts=True)
    assert torch.allclose(p0["out_fp32"] + p1["out_fp32"], parts["out_fp32"], rtol=1e-5, atol=1e-6)


# ------------------------------------------------------------ C ABI, host side
def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "msk_moe.h")).read()
    return sorted(set(re.findall(r"^int (msk_\w+)\(", text, flags=re.M)))


def test_library_exports_every_declared_symbol():
    from muse_moe_w4a16 import _lib

    lib = _lib.load()
    declared = _declared_symbols()
    assert len(declared) >= 14
    for name in declared:
        assert hasattr(lib, name), name
    assert sorted(_lib.SIGNATURES) == declared  # the binding table and the header agree


def test_host_side_validation_rejects_bad_arguments():
    from muse_moe_w4a16 import _lib

    lib = _lib.load()
    good = dict(hidden=512, inter=256, n_experts=8, local_start=0, local_count=8, top_k=2, max_tokens=4)
    cfg = _lib.MskMoeCfg(**good)
    a, b = ctypes.c_size_t(), ctypes.c_size_t()
    assert lib.msk_moe_packed_bytes(ctypes.byref(cfg), ctypes.byref(a), ctypes.byref(b)) == 0
    assert a.value == 8 * (2 * 256 // 128) * (512 // 256) * 18432 and b.value == 8 * (512 // 128) * 1 * 18432
    assert lib.msk_moe_packed_bytes(None, ctypes.byref(a), ctypes.byref(b)) == -1
    for bad in (dict(hidden=500), dict(inter=128), dict(top_k=0), dict(top_k=17), dict(local_count=0),
                dict(local_count=300), dict(n_experts=600), dict(token_tile=8), dict(token_tile=48),
                dict(decode_path=5), dict(decode_path=-1)):
        c = _lib.MskMoeCfg(**{**good, **bad})
        assert lib.msk_moe_packed_bytes(ctypes.byref(c), ctypes.byref(a), ctypes.byref(b)) == -2, bad
    c = _lib.MskMoeCfg(**{**good, "local_start": 4})
    assert lib.msk_moe_packed_bytes(ctypes.byref(c), ctypes.byref(a), ctypes.byref(b)) == -5
    ws = ctypes.c_size_t()
    assert lib.msk_moe_workspace_bytes(ctypes.byref(cfg), ctypes.byref(ws)) == 0 and ws.value > 4 * 2 * 512 * 4
    # forward: NULL pointers, too many tokens, undersized workspace are refused before any launch
    p = ctypes.c_void_p(0)
    assert lib.msk_moe_forward(ctypes.byref(cfg), p, p, p, p, p, p, p, p, p, p, 0, 1, p) == -1
    fake = ctypes.c_void_p(4096)
    assert lib.msk_moe_forward(ctypes.byref(cfg), fake, fake, fake, fake, None, fake, fake, fake, fake, fake,
                               ws.value, 5, None) == -6
    assert lib.msk_moe_forward(ctypes.byref(cfg), fake, fake, fake, fake, None, fake, fake, fake, fake, fake,
                               16, 4, None) == -4
    odd = ctypes.c_void_p(4100)
    assert lib.msk_moe_forward(ctypes.byref(cfg), odd, fake, fake, fake, None, fake, fake, fake, fake, fake,
                               ws.value, 4, None) == -3
    plan = (ctypes.c_int * 4)()
    assert lib.msk_moe_plan(ctypes.byref(cfg), 4, plan) == 0 and plan[0] in (16, 32, 64, 128)


def _pieces(lib, n_base, nst, shares, mode, cta, heavy=0, skip=0):
    cap = 4096
    buf = (ctypes.c_int * (6 * cap))()
    n = ctypes.c_int()
    assert lib.msk_moe_share_pieces(n_base, nst, shares, mode, cta, heavy, skip, buf, cap, ctypes.byref(n)) == 0
    return [tuple(buf[6 * i:6 * i + 6]) for i in range(n.value)]


@pytest.mark.parametrize("n_base,nst,shares", [(96, 16, 148), (128, 6, 148), (600, 16, 148), (3, 28, 148), (1, 1, 7),
                                               (0, 16, 148), (37, 5, 5), (224, 8, 148), (50, 2, 1)])
def test_flat_shares_cover_every_stage_once_and_name_their_pieces(n_base, nst, shares):
    """The work distribution of the GEMM kernels (host twin of the device code): with flat shares (full
    rounds of whole units, then the last full round and the left-over units cut into equal shares of
    stages; nothing is cut when there are fewer units than CTAs)
    every (unit, stage) item belongs to exactly one CTA, shares differ by at most one item, a cut unit's
    pieces sit in consecutive CTAs in ascending K order, each in a slot of its own, and the first / last
    owner every piece computes is the CTA that really holds the unit's first / last stage."""
    from muse_moe_w4a16 import _lib

    lib = _lib.load()
    seen = {}
    sizes = []
    slots = set()
    for c in range(shares):
        pcs = _pieces(lib, n_base, nst, shares, 1, c)
        sizes.append(sum(k1 - k0 for _, k0, k1, *_ in pcs))
        for base, k0, k1, slot, first, last in pcs:
            assert 0 <= k0 < k1 <= nst
            for ks in range(k0, k1):
                assert (base, ks) not in seen
                seen[(base, ks)] = c
            if slot >= 0:
                assert slot not in slots and slot // 2 == c
                slots.add(slot)
            else:
                assert (k0, k1) == (0, nst)
    assert len(seen) == n_base * nst
    if n_base >= shares:
        assert max(sizes) - min(sizes) <= 1
    else:                       # fewer units than CTAs: nothing is cut
        assert set(sizes) <= {0, nst} and not slots
    for c in range(shares):
        for base, k0, k1, slot, first, last in _pieces(lib, n_base, nst, shares, 1, c):
            assert first == seen[(base, 0)] and last == seen[(base, nst - 1)]
            owners = [seen[(base, ks)] for ks in range(nst)]
            assert owners == sorted(owners) and first <= min(owners) and max(owners) <= last
            # every share between the first and the last owner either holds a piece of the unit or has an empty
            # share of the tail (the units left over after the full rounds of whole units)
            tail_first = n_base if n_base < shares else (n_base // shares - 1) * shares
            tail_items = (n_base - tail_first) * nst
            empty = lambda c: tail_items * (c + 1) // shares == tail_items * c // shares
            assert all(c in owners or empty(c) for c in range(first, last + 1))


def test_whole_unit_mode_gives_every_unit_to_one_cta():
    from muse_moe_w4a16 import _lib

    lib = _lib.load()
    n_base, nst, shares = 301, 16, 148
    got = []
    for c in range(shares):
        for base, k0, k1, slot, first, last in _pieces(lib, n_base, nst, shares, 0, c):
            assert (k0, k1, slot) == (0, nst, -1)
            got.append(base)
    assert sorted(got) == list(range(n_base))


@pytest.mark.parametrize("n0,nst0,n1,nst1,shares", [(600, 16, 800, 6, 148), (96, 16, 128, 6, 148), (1356, 16, 1808, 6, 148),
                                                     (300, 28, 100, 8, 148), (5, 2, 3, 1, 4)])
def test_skewed_dealing_of_the_second_phase_balances_both_phases(n0, nst0, n1, nst1, shares):
    """One launch for both GEMMs: the CTAs that hold one more gate/up unit are left out of the first
    rounds of down units. Every down unit still goes to exactly one CTA, each CTA takes its units in
    ascending order, and the largest total (in K stages) is no larger than with plain round-robin."""
    from muse_moe_w4a16 import _lib

    lib = _lib.load()
    heavy = n0 % shares if n0 >= shares else 0   # the rule of the kernel (phase1_skew)
    skip = (nst0 + nst1 // 2) // nst1 if heavy else 0
    load0 = [len(_pieces(lib, n0, nst0, shares, 0, c)) * nst0 for c in range(shares)]
    got, skewed, plain = [], [], []
    for c in range(shares):
        mine = [b for b, *_ in _pieces(lib, n1, nst1, shares, 0, c, heavy, skip)]
        assert mine == sorted(mine)
        got += mine
        skewed.append(load0[c] + len(mine) * nst1)
        plain.append(load0[c] + len(_pieces(lib, n1, nst1, shares, 0, c)) * nst1)
    assert sorted(got) == list(range(n1))
    assert max(skewed) <= max(plain)


def test_plan_is_a_function_of_the_configuration_only():
    """Token tile, path and grid follow from the shapes and the token count (never from the device:
    the default grid is a constant): up to 8 tokens the whole step is one launch, beyond that the narrow
    token tiles run both GEMMs in one launch behind the sort (path 4), the wide tiles the chain."""
    from muse_moe_w4a16 import _lib

    lib = _lib.load()
    plan = (ctypes.c_int * 4)()
    cfg = _lib.MskMoeCfg(hidden=4096, inter=1536, n_experts=128, local_start=0, local_count=128, top_k=8, max_tokens=8192)
    want = {1: (16, 0, 0, 148), 8: (16, 0, 0, 148), 9: (16, 4, 0, 148), 32: (16, 4, 0, 148), 64: (16, 4, 0, 148),
            256: (64, 1, 0, 148), 8192: (128, 1, 0, 148)}
    for T, w in want.items():
        assert lib.msk_moe_plan(ctypes.byref(cfg), T, plan) == 0
        assert tuple(plan) == w, (T, tuple(plan))
    cfg.decode_path = 2
    cfg.flat_shares = 1
    assert lib.msk_moe_plan(ctypes.byref(cfg), 8, plan) == 0 and tuple(plan) == (16, 2, 1, 148)
    cfg.decode_path = 3
    assert lib.msk_moe_plan(ctypes.byref(cfg), 32, plan) == 0 and tuple(plan) == (16, 0, 0, 148)
    cfg.decode_path = 4
    assert lib.msk_moe_plan(ctypes.byref(cfg), 190, plan) == 0 and tuple(plan) == (16, 4, 0, 148)
    cfg.token_tile = 32
    assert lib.msk_moe_plan(ctypes.byref(cfg), 190, plan) == 0 and tuple(plan) == (32, 4, 0, 148)
    cfg.token_tile = 0
    assert lib.msk_moe_plan(ctypes.byref(cfg), 256, plan) == 0 and tuple(plan) == (64, 1, 0, 148)   # wide tile: the chain
    cfg.decode_path = 1
    cfg.num_ctas = 37
    assert lib.msk_moe_plan(ctypes.byref(cfg), 8, plan) == 0 and tuple(plan) == (16, 1, 1, 37)
    assert lib.msk_moe_plan(ctypes.byref(cfg), 64, plan) == 0 and tuple(plan) == (16, 1, 0, 37)


@pytest.mark.parametrize("asked,T,plan", [({}, 28, (16, 0)), ({}, 29, (64, 0)), (dict(flat_shares=1), 29, (16, 1)), (dict(flat_shares=1), 48, (16, 1)),
                                          (dict(flat_shares=1), 49, (64, 1)), (dict(stop_after=1), 48, (16, 0)), (dict(stop_after=3), 49, (64, 0)),
                                          (dict(decode_path=1), 48, (16, 0))])
def test_a_form_that_is_asked_for_keeps_the_narrow_tile(asked, T, plan):
    """From 7 rows an expert on the default tile is 64; paths, flat shares and parts of the step, asked for, keep the 16-token tile to 12."""
    from muse_moe_w4a16 import _lib

    cfg = _lib.MskMoeCfg(**dict(dict(hidden=2048, inter=1024, n_experts=16, local_start=0, local_count=16, top_k=4, max_tokens=64), **asked))
    out = (ctypes.c_int * 4)()
    assert _lib.load().msk_moe_plan(ctypes.byref(cfg), T, out) == 0
    assert (out[0], out[2]) == plan


def _few_fits(T, inputs=0, **shape):
    from muse_moe_w4a16 import _lib

    cfg = _lib.MskMoeCfg(**dict(dict(local_start=0, max_tokens=64), **shape))
    fits = ctypes.c_int(-1)
    assert _lib.load().msk_moe_few_fits(ctypes.byref(cfg), T, inputs, ctypes.byref(fits)) == 0
    return bool(fits.value)


@pytest.mark.parametrize("T,k,inputs", [(1, 1, 0), (3, 8, 0), (1, 16, 1), (4, 16, 2), (4, 16, 3)])
def test_few_token_kernel_numbers_its_tiles_exactly(T, k, inputs):
    """moe_few_kernel finds the tile of gate/up unit u as the high half of u * ceil(2^32 / (I / 8)): where a step is
    accepted that is u // (I / 8) for every unit it can have (at most one tile per routed row), and wider experts go to
    another kernel. Sizes: the usual ones, around the line for 64 rows, and around those for 24, 16 and one."""
    widths = [256, 1536, 4096, 8192, 14336, 28672] + [256 * i for i in range(200, 280)] + [256 * i for i in range(410, 440)] \
        + [256 * i for i in range(500, 540)] + [256 * i for i in range(2040, 2060)]
    seen = set()
    for width in widths:
        fits = _few_fits(T, inputs, hidden=256, inter=width, n_experts=64, local_count=64, top_k=k)
        n = width // 8
        inv = -(-2 ** 32 // n)
        last = np.arange(1, T * k + 1, dtype=object) * n - 1          # the last unit of every tile goes wrong first
        exact = all((int(u) * inv) >> 32 == int(u) // n for u in last)
        assert fits == exact or (not fits and width > 53000), width
        seen.add(fits)
    assert True in seen and (k * T < 64 or False in seen)


def test_configuration_struct_is_the_documented_one():
    """A host compiled against the documented struct must hand over every byte the library reads: the same fields in
    the same order in the header, the Python binding and the integration guide."""
    from muse_moe_w4a16 import _lib

    header = open(os.path.join(ROOT, "include", "msk_moe.h")).read()
    body = re.sub(r"/\*.*?\*/", "", header[header.index("typedef struct MskMoeCfg"):header.index("} MskMoeCfg;")], flags=re.S)
    fields = re.findall(r"(?:int32_t|float)\s+(\w+);", body)
    assert fields == [n for n, _ in _lib.MskMoeCfg._fields_]
    guide = open(os.path.join(ROOT, "INTEGRATION.md")).read()
    stub = guide[guide.index("class MskMoeCfg"):guide.index("lib = ctypes.CDLL")]
    assert re.findall(r'"(\w+)"', stub) == fields


@pytest.mark.parametrize("shape,takes", [      # tokens up to which the kernel is taken: plain, rows in host memory, pre-norm
    (dict(hidden=4096, inter=1536, n_experts=128, local_count=128, top_k=8), (3, 2, 4)),     # eight local routes a token
    (dict(hidden=4096, inter=4096, n_experts=256, local_count=32, top_k=8), (3, 3, 6)),      # one
    (dict(hidden=7168, inter=2048, n_experts=256, local_count=32, top_k=8), (3, 3, 4)),      # one, longer rows
    (dict(hidden=2048, inter=1024, n_experts=64, local_count=64, top_k=4), (3, 3, 6))])      # four
def test_few_token_kernel_is_taken_where_it_was_measured_faster(shape, takes):
    for inputs, most in zip((0, 4, 2), takes):
        for given in (0, 1):
            assert [T for T in range(1, 9) if _few_fits(T, inputs | given, **shape)] == list(range(1, most + 1)), (inputs, given)


def test_few_token_kernel_leaves_normed_rows_in_host_memory_to_another():
    """With the pre-expert norm every CTA of moe_few_kernel reads whole token rows: not over PCIe."""
    shape = dict(hidden=4096, inter=1536, n_experts=128, local_count=128, top_k=8)
    assert _few_fits(1, 2, **shape) and _few_fits(1, 4, **shape) and _few_fits(1, 5, **shape)
    assert not any(_few_fits(T, 2 | 4 | given, **shape) for T in (1, 2, 6) for given in (0, 1))


_ONE = dict(hidden=4096, inter=1536, n_experts=128, local_count=128, top_k=8)
_RANK = dict(hidden=4096, inter=4096, n_experts=256, local_count=32, top_k=8)


@pytest.mark.parametrize("shape,norms,taken", [      # ranges of token counts: with no norm 0, the post-expert one 1, the pre-expert one 2, both 3
    (_ONE, 0, [(6, 192)]), (_ONE, 1, [(4, 192)]), (_ONE, 2, [(4, 192)]), (_ONE, 3, [(4, 192)]),
    (_RANK, 0, [(20, 384)]), (_RANK, 1, [(4, 8), (20, 384)]), (_RANK, 2, [(20, 384)]), (_RANK, 3, [(4, 8), (20, 384)]),
    (dict(_ONE, inter=1280), 0, []), (dict(_ONE, inter=1280), 1, []),
    (dict(_ONE, hidden=2048, n_experts=64, local_count=64, top_k=4), 0, []),                   # 340 MB in all
    (dict(_ONE, hidden=2048, n_experts=64, local_count=64, top_k=4), 1, [(4, 8)]),
    (dict(_ONE, hidden=2048, n_experts=64, local_count=64, top_k=4), 2, [(9, 192)]),
    (dict(_ONE, hidden=2048, inter=2048, n_experts=64, local_count=64, top_k=4), 0, []),       # 453 MB
    (dict(_ONE, hidden=2048, inter=2304, n_experts=64, local_count=64, top_k=4), 0, [(37, 192)]),   # 510 MB
    (dict(_ONE, n_experts=8, local_count=8, top_k=2), 0, [(6, 48)]),
    (dict(_ONE, num_ctas=256), 0, []), (dict(_ONE, token_tile=16), 0, []), (dict(_ONE, decode_path=1), 0, []), (dict(_ONE, decode_path=4), 0, []),
    (dict(_ONE, flat_shares=1), 0, []), (dict(_ONE, stop_after=1), 0, []), (dict(_ONE, hidden=8192), 0, [(6, 192)])])
def test_fp4_kernel_is_taken_where_it_was_measured_faster(shape, norms, taken):
    """Both sides of every line of the rule, and never where a tile, a path or a part of the step was asked for."""
    from muse_moe_w4a16 import _lib

    cfg = _lib.MskMoeCfg(**dict(dict(local_start=0, max_tokens=512), **shape))
    got = []
    for T in range(1, 513):
        takes = ctypes.c_int(-1)
        assert _lib.load().msk_moe_nvf4_takes(ctypes.byref(cfg), T, norms, ctypes.byref(takes)) == 0
        if takes.value:
            got.append(T)
    assert got == [T for a, b in taken for T in range(a, b + 1)]


_SMALL = dict(hidden=2048, inter=1024, n_experts=64, local_count=64, top_k=4)
_GIVEN, _PRE, _HOST_X, _POST, _HOST_ROUTES = 1, 2, 4, 8, 16                              # inputs of msk_moe_step_form
_ONE_LAUNCH, _CHAIN, _FOLDED, _BOTH, _FEW, _NVF4 = 0, 1, 2, 4, 5, 6      # what it answers


@pytest.mark.parametrize("shape,inputs,forms", [     # (first token count, form), each up to the next one
    (_SMALL, 0, [(1, _FEW), (4, _ONE_LAUNCH), (9, _BOTH)]), (_SMALL, _GIVEN, [(1, _FEW), (4, _ONE_LAUNCH), (9, _BOTH)]),
    (_SMALL, _POST, [(1, _FEW), (4, _BOTH)]), (_SMALL, _HOST_X, [(1, _FEW), (4, _BOTH)]), (_SMALL, _HOST_X | _POST, [(1, _FEW), (4, _BOTH)]),
    (_SMALL, _PRE, [(1, _FEW), (7, _FOLDED), (9, _CHAIN), (113, _BOTH)]),          # (narrow tiles to 7 rows an expert, row copy in front of them)
    (_SMALL, _PRE | _POST, [(1, _FEW), (7, _CHAIN), (113, _BOTH)]),
    # both norms: the chain from five tokens on, with more than two local routes a token, two of 40 MB, one behind the top-k of 128 experts
    (dict(_SMALL, local_count=16), _PRE | _POST, [(1, _FEW), (7, _FOLDED), (9, _CHAIN), (113, _BOTH)]),
    (dict(_SMALL, local_count=32), _PRE | _POST, [(1, _FEW), (7, _CHAIN), (113, _BOTH)]),
    (dict(_SMALL, local_count=32, inter=768), _PRE | _POST, [(1, _FEW), (7, _FOLDED), (8, _CHAIN), (113, _BOTH)]),
    (dict(_SMALL, hidden=7168, n_experts=256, local_count=32, top_k=8), _PRE | _POST, [(1, _FEW), (5, _CHAIN), (225, _BOTH)]),
    (dict(_SMALL, hidden=7168, n_experts=256, local_count=32, top_k=8), _GIVEN | _PRE | _POST, [(1, _FEW), (5, _FOLDED), (9, _CHAIN), (225, _BOTH)]),
    # rows in host memory, routes on the device or there as well
    (_SMALL, _HOST_X | _PRE | _POST, [(1, _FOLDED), (9, _CHAIN), (113, _BOTH)]), (_SMALL, _HOST_X | _PRE, [(1, _FOLDED), (9, _CHAIN), (113, _BOTH)]),
    (dict(_SMALL, top_k=8), _HOST_X | _PRE | _POST, [(1, _FOLDED), (5, _CHAIN), (57, _BOTH)]),
    (_SMALL, _HOST_X | _HOST_ROUTES | _PRE, [(1, _FOLDED), (3, _CHAIN), (113, _BOTH)]),
    (dict(_SMALL, local_count=32), _HOST_X | _HOST_ROUTES | _GIVEN | _PRE | _POST, [(1, _FOLDED), (9, _CHAIN), (113, _BOTH)]),
    (_ONE, 0, [(1, _FEW), (4, _ONE_LAUNCH), (6, _NVF4), (193, _BOTH)]), (_ONE, _POST, [(1, _FEW), (4, _NVF4), (193, _BOTH)]),
    (_ONE, _HOST_X, [(1, _FEW), (3, _BOTH), (6, _NVF4), (193, _BOTH)]),
    (_RANK, 0, [(1, _FEW), (4, _ONE_LAUNCH), (9, _BOTH), (20, _NVF4), (385, _BOTH)]),
    (_RANK, _PRE | _POST, [(1, _FEW), (7, _NVF4), (9, _CHAIN), (20, _NVF4), (385, _BOTH)]),
    (dict(_SMALL, decode_path=3), _POST, [(1, _FEW), (4, _ONE_LAUNCH), (33, _CHAIN), (193, _BOTH)]),
    (dict(_SMALL, decode_path=3), _PRE | _POST, [(1, _FEW), (7, _FOLDED), (33, _CHAIN), (193, _BOTH)]),
    (dict(_SMALL, decode_path=2), _POST, [(1, _FOLDED), (33, _CHAIN), (193, _BOTH)]),
    (dict(_SMALL, decode_path=1), _POST, [(1, _CHAIN)]), (dict(_SMALL, decode_path=4), _POST, [(1, _BOTH)]),
    (dict(_SMALL, num_ctas=256), 0, [(1, _FOLDED), (9, _CHAIN), (641, _BOTH)])])
def test_step_form_names_what_a_step_runs_in(shape, inputs, forms):
    """Both sides of every line between the forms, by the function that launches them: four tokens with the post-expert norm, rows in host
    memory, the end of the narrow tile (7 rows an expert, 12 where a path is asked for), the FP4 and the few-token kernel."""
    from muse_moe_w4a16 import _lib

    cfg = _lib.MskMoeCfg(**dict(dict(local_start=0, max_tokens=1024), **shape))
    want = {}
    for first, form in forms:
        want.update({T: form for T in range(first, 1025)})
    got = {}
    for T in range(1, 1025):
        form = ctypes.c_int(-1)
        # (rows in host memory make a difference up to eight tokens only)
        assert _lib.load().msk_moe_step_form(ctypes.byref(cfg), T, inputs & ~(_HOST_X | _HOST_ROUTES if T > 8 else 0), ctypes.byref(form)) == 0
        got[T] = form.value
    assert got == want, [(T, got[T], want[T]) for T in got if got[T] != want[T]][:5]


def test_workspace_init_covers_every_control_word():
    """msk_moe_workspace_init zeroes everything in front of `inter`: the status word, the sort tables,
    both ticket regions, the control words of the few-token paths (token tickets, grid and tile
    counters), the per-CTA counts of the multi-CTA sort and the tile counters of the hand-over between the
    two GEMM launches must all lie there."""
    from muse_moe_w4a16 import _lib

    lib = _lib.load()
    cfg = _lib.MskMoeCfg(hidden=4096, inter=1536, n_experts=128, local_start=0, local_count=128, top_k=8, max_tokens=256)
    base = 1 << 20

    def off(which):
        p = ctypes.c_void_p()
        assert lib.msk_moe_workspace_view(ctypes.byref(cfg), ctypes.c_void_p(base), which, ctypes.byref(p)) == 0
        return p.value - base

    inter = off(4)
    pairs = max(1536 // 128, 4096 // 256)
    tiles = 256 * 8 // 16 + 128
    for which, nbytes in ((0, 128 * 4), (1, 129 * 4), (2, 2048 * 4), (3, 2048 * 4), (7, 2 * tiles * pairs * 4),
                          (8, 8192), (9, 64 * 256 * 4), (10, 2 * tiles * 4)):
        assert 256 <= off(which) and off(which) + nbytes <= inter, which
    ws = ctypes.c_size_t()
    assert lib.msk_moe_workspace_bytes(ctypes.byref(cfg), ctypes.byref(ws)) == 0
    assert ws.value < 200 << 20      # the pieces of cut units take two slots per CTA, not a split-K buffer per unit


def test_workspace_has_room_of_its_own_for_split_rows_only_where_they_need_it():
    """The FP4 kernel's split rows lie where the F16 rows and the pieces of cut units would: nothing more for a large capacity, the
    rest of them for a small one, and nothing where a form is asked for whose steps never take it."""
    from muse_moe_w4a16 import _lib

    lib = _lib.load()

    def size(**shape):
        ws = ctypes.c_size_t()
        assert lib.msk_moe_workspace_bytes(ctypes.byref(_lib.MskMoeCfg(**dict(dict(local_start=0), **shape))), ctypes.byref(ws)) == 0
        return ws.value

    for shape in (_ONE, _RANK, dict(_RANK, hidden=7168, inter=2048)):
        for form in (dict(token_tile=16), dict(decode_path=1), dict(flat_shares=1), dict(stop_after=1)):
            assert size(max_tokens=8192, **shape) == size(max_tokens=8192, **dict(shape, **form))
            assert size(max_tokens=64, **shape) > size(max_tokens=64, **dict(shape, **form))
        # images: 15,744 bytes for eight rows x 256 K, at most a group more per expert than full ones
        H, I, rows = shape["hidden"], shape["inter"], 64 * shape["top_k"]
        groups = shape["local_count"] + (rows - shape["local_count"]) // 8
        more = size(max_tokens=64, **shape) - size(max_tokens=64, token_tile=16, **shape)
        assert more < groups * (H + I) // 256 * 15744
    assert size(max_tokens=8192, **_ONE) < 1.853e9


def test_module_refuses_cpu_tensors():
    import muse_moe_w4a16 as moe
    from muse_moe_w4a16 import inputs

    w = inputs.make_weights(256, 256, 2, 0, "cpu")
    with pytest.raises(RuntimeError, match="CUDA"):
        moe.prepare(w)


def test_oracle_pre_expert_norm_is_the_norm_in_front_of_the_step():
    """pre_expert_norm follows muse_decode_layer/py/04_triton_kernels.py:556-568 (RMS over the row,
    eps 1e-5, times 1 + g, one rounding to bf16), and moe_forward with weights["pre_norm_w"] equals
    moe_forward on the normed rows."""
    from muse_moe_w4a16 import inputs
    from oracle import moe_oracle as orc

    H, I, E, k, T = 256, 256, 4, 2, 5
    w = inputs.make_weights(H, I, E, 3, "cpu", post_norm=True)
    g = torch.Generator().manual_seed(2)
    x = (torch.randn((T, H), generator=g) * 2.0).to(torch.bfloat16)
    gw = (torch.randn((H,), generator=g) * 0.1).to(torch.bfloat16)
    xn = orc.pre_expert_norm(x, gw)
    xf = x.float()
    want = xf / torch.sqrt((xf * xf).sum(-1, keepdim=True) / H + 1e-5) * (1.0 + gw.float())
    assert xn.dtype == torch.bfloat16
    assert float((xn.float() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    ids, tw = orc.route_topk(torch.randn((T, E), generator=g), k)
    a = orc.moe_forward(x, ids, tw, dict(w, pre_norm_w=gw))
    b = orc.moe_forward(xn, ids, tw, w)
    assert torch.equal(a, b)


# ------------------------------- vectors produced by the reference's Triton kernels on a CPU
def _bf16(a):
    return torch.from_numpy(a.astype(np.int16)).view(torch.bfloat16)


def test_routing_matches_reference_route_split():
    """ids, local ids and weights of the reference's `_route_split` (sigmoid(logit / sqrt(32)) + bias,
    eight rounds of arg-max, ties to the lowest index), on logits that hold exact ties."""
    logits, bias = torch.from_numpy(GOLD["rs_logits"]), torch.from_numpy(GOLD["rs_bias"])
    ids, w = orc.route_topk(logits, 8, "sigmoid_bias", bias)
    assert np.array_equal(ids.numpy(), GOLD["rs_ids"])
    assert np.allclose(w.numpy(), GOLD["rs_w"], rtol=2e-6, atol=1e-8)
    # the constructed ties are there and went to the lower index
    assert list(GOLD["rs_ids"][1]) == sorted(GOLD["rs_ids"][1].tolist(), key=lambda e: (-float(bias[e]), e))
    assert not np.isin(GOLD["rs_ids"], np.arange(200, 208)).any() or np.isin(GOLD["rs_ids"], np.arange(8, 16)).any()
    ls = int(GOLD["rs_local_start"][0])
    assert np.array_equal(orc.local_ids(ids, ls, 32).numpy(), GOLD["rs_lids"])
    # the stable sort drops exactly the entries the reference marks -1
    cnt, off, perm, inv = orc.sort_routes(GOLD["rs_ids"], ls, 32)
    assert np.array_equal(inv >= 0, GOLD["rs_lids"].reshape(-1) >= 0)
    assert np.array_equal(GOLD["rs_lids"].reshape(-1)[perm], np.sort(GOLD["rs_lids"].reshape(-1)[perm], kind="stable"))


def _trunc_bf16(f):
    """FP32 -> BF16 by dropping the low 16 bits: how Triton's CPU interpreter converts (compiled for
    a GPU the same kernels round to nearest even, as the oracle and the CUDA path do). The golden
    BF16 outputs are therefore compared with the truncated FP32 values of the oracle, which pins the
    FP32 arithmetic in front of the rounding."""
    return (f.contiguous().view(torch.int32) & -65536).view(torch.float32)


def test_pre_expert_norm_matches_reference_route_split():
    """The expert input the reference's routing kernel stores: x * rsqrt(sum(x^2)/H + 1e-5) * (1 + g)."""
    f = orc.pre_expert_norm(_bf16(GOLD["rs_pooled"]), _bf16(GOLD["rs_gpre"]), return_fp32=True)
    want = _bf16(GOLD["rs_x"]).float()
    same = _trunc_bf16(f) == want
    # a row's sum of 4096 squares is taken in another order by the two programs: allow the last FP32 bit
    # of the scale to move a value across a BF16 boundary on a handful of elements
    assert float(same.float().mean()) > 0.999
    assert bool(((f - want).abs() <= 2.0 ** -7 * want.abs() + 1e-30).all())
    rn = orc.pre_expert_norm(_bf16(GOLD["rs_pooled"]), _bf16(GOLD["rs_gpre"]))
    assert rn.dtype == torch.bfloat16 and bool(((rn.float() - f).abs() <= 2.0 ** -8 * f.abs()).all())


def test_combine_matches_reference_pexp_norm_sum():
    """Post-expert norm (1 + w first, RMS over the row, eps 1e-8) times the routing weight, summed in
    slot order over the slots with a local expert; a token without one is zero."""
    y = _bf16(GOLD["pn_y"]).float()
    pw = _bf16(GOLD["pn_w"]).float()
    s, lid = torch.from_numpy(GOLD["pn_s"]), torch.from_numpy(GOLD["pn_ids"])
    T, K = lid.shape
    inv = torch.where(lid >= 0, torch.arange(T * K, dtype=torch.int32).view(T, K), torch.full_like(lid, -1))
    out = orc.combine_rows(y * (1.0 + pw), inv, s, True, 1e-8)
    want = _bf16(GOLD["pn_out"]).float()
    assert float(want[2].abs().max()) == 0.0 and float(out[2].abs().max()) == 0.0
    same = _trunc_bf16(out) == want
    assert float(same.float().mean()) > 0.995          # the rest straddle a BF16 boundary in their last FP32 bits
    assert float((out - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())


def test_timeline_stamp_slots_follow_the_kernel_enum():
    """muse_moe_w4a16.timeline names the kernels' trace slots by number; the numbers must be the positions
    of the TR_* enumerators in csrc/gemm.cuh."""
    import re

    from muse_moe_w4a16 import timeline

    src = open(os.path.join(ROOT, "muse-spark-kernels_b200", "csrc", "gemm.cuh")).read()
    body = re.search(r"enum\s*:\s*int\s*\{\s*(TR_START\s*=\s*0.*?)\};", src, re.S).group(1)
    names = [n.strip().split("=")[0].strip() for n in body.replace("\n", " ").split(",") if n.strip()]
    slots = {n[3:]: i for i, n in enumerate(names)}
    assert len(slots) <= 16                      # 16 stamps per CTA in the workspace
    for name, slot in timeline.STAMPS:
        assert slots[name] == slot, name
    assert {n for n, _ in timeline.STAMPS} == set(slots)


def _kernel_body(name, kernel):
    """Source text of a kernel, comments and string literals left out."""
    src = open(os.path.join(ROOT, "muse-spark-kernels_b200", "csrc", name)).read()
    src = re.sub(r"//[^\n]*", "", src)
    at = src.index("{", src.index(")", src.index(kernel + "(")))
    depth = 0
    for i in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[at:i + 1]
    raise AssertionError(kernel)


def test_few_token_kernel_gives_up_a_warp_at_a_time():
    """A bounded wait of moe_few_kernel that runs out must send the whole warp the same way: the kernel body
    waits on its barriers and mailboxes through the warp-wide forms only, and those end in a warp vote or a
    broadcast."""
    body = _kernel_body("few.cuh", "moe_few_kernel")
    waits = re.findall(r"\b\w*mbar_(?:try_)?wait\w*|\b\w*mail_\w+", body)
    assert len(waits) >= 5 and set(waits) == {"warp_mbar_wait", "warp_mail_post"}
    assert "__all_sync" in _kernel_body("few.cuh", "bool warp_mbar_wait")
    assert "__shfl_sync" in _kernel_body("few.cuh", "bool warp_mail_post").split("return")[-1]


def test_kernels_read_other_ctas_rows_behind_a_barrier():
    """Rows that other CTAs wrote are read by all lanes after lane 0 acquired their counter: a shuffle orders no
    memory, so the wait ends in __syncwarp() (the one of the norm sums, by a single thread, in __syncthreads())."""
    body = _kernel_body("few.cuh", "moe_few_kernel")
    waits = [m.end() for m in re.finditer(r"\bwarp_counter_wait\(", body)]
    assert len(waits) == 2
    assert re.findall(r"\bgrid_counter_spin\([^;]*;\s*\}\s*(\w+)", body) == ["__syncthreads"] * body.count("grid_counter_spin(")
    tail = _kernel_body("few.cuh", "bool warp_counter_wait")
    assert tail.index("__shfl_sync") < tail.index("__syncwarp")
    gather = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "muse-spark-kernels_b200", "csrc", "gemm_gather.inl")).read())
    assert re.findall(r"go = __shfl_sync\([^;]*;\s*(\w+)", gather) == ["__syncwarp"]


@pytest.mark.parametrize("name,kernel,written", [("route_sort.cuh", "sort_multi_scatter_kernel", ("ids", "blk")),
                                                 ("route_sort.cuh", "sort_multi_count_kernel", ("logits",)),
                                                 ("route_sort.cuh", "route_sort_kernel", ("logits",)),
                                                 ("route_sort.cuh", "route_topk_kernel", ("logits",)),
                                                 ("route_sort.cuh", " sort_kernel", ("ids",)),
                                                 ("msk_moe.cu", "combine_norm_kernel", ("y", "inv", "tw")),
                                                 ("msk_moe.cu", "combine_cols_kernel", ("y", "inv", "tw"))])
def test_what_the_launch_before_writes_is_read_coherently(name, kernel, written):
    """A kernel started by programmatic launch is there while its predecessor still writes: what that one writes must
    not go through the read-only path, which __ldg asks for and const __restrict__ allows."""
    src = open(os.path.join(ROOT, "muse-spark-kernels_b200", "csrc", name)).read()
    at = re.search(kernel + r"\((const)", src).start()
    args = src[at:src.index(")", at)]
    for arg in written:
        assert not re.search(r"__restrict__ " + arg + r"\b", args), arg
        assert not re.search(r"__ldg\([^;]*\b" + arg + r"\b", _kernel_body(name, kernel)), arg
