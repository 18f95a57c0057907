"""Batch sizes and row widths on both sides of every line at which the whole-layer entries change their kernels or tile widths,
against the CPU oracle: token tiles of 16 / 32 / 64 / 128 columns, ragged last row tiles, one or two pairs per GEMV entry, the
decode entry's step to the GEMM, the tiled router and its padding for every row width."""
import numpy as np
import pytest
import torch

import oracle
from chimere_b200 import configs, formats
from chimere_b200.layer import (MoeScratch, MoeWeightsPrefill, MoeWeightsTiled, forward_moe, forward_moe_host, forward_moe_prefill, forward_moe_residual_norm,
                                route_only)
from parity_util import check_rows, oracle_on_gpu_routing

pytestmark = pytest.mark.gpu
Q4, Q8, IQ3 = configs.QWEN_Q4_0, configs.QWEN_Q8_0, configs.QWEN_IQ3S


def _check(cfg, T, prefill):
    raw = configs.make_layer(cfg, device="cuda")
    tiled = MoeWeightsTiled(raw)
    x = configs.make_input(cfg, T, device="cuda")
    sc = MoeScratch(tiled, T)
    y = forward_moe_prefill(tiled, MoeWeightsPrefill(raw), sc, x) if prefill else forward_moe(tiled, sc, x)
    torch.cuda.synchronize()
    assert sc.status() == 0
    idx = sc.topk_indices(T).cpu().numpy()
    o = oracle_on_gpu_routing(raw.to("cpu"), x.cpu().numpy(), idx)
    assert np.array_equal(sc.router_logits(T).cpu().numpy(), o["logits"])
    assert np.array_equal(sc.x_q8(T).cpu().numpy(), o["x_q8"])
    perm, offs = oracle.permute(idx, cfg.E)
    assert np.array_equal(sc.perm(T).cpu().numpy(), perm) and np.array_equal(sc.offsets().cpu().numpy(), offs)
    check_rows(y.cpu().numpy(), o["y"])


# one expert that every token uses: the token count is the tile's column count
@pytest.mark.parametrize("base", [Q4, IQ3, Q8], ids=lambda c: c.name)
@pytest.mark.parametrize("T", [1, 15, 16, 17, 32, 33, 64, 65, 127, 128, 129, 161])
def test_token_tile_widths(base, T):
    _check(configs.scaled(base, E=1, top_k=1, H=512, F=256, F_s=256, zipf_bias=False), T, prefill=True)


# 32-row tiles that do not fill the last 128-row tile, K that does not fill the last stage of four blocks
@pytest.mark.parametrize("kw", [dict(F=96, F_s=160, H=384), dict(F=160, F_s=32, H=128), dict(F=224, F_s=96, H=640)], ids=str)
@pytest.mark.parametrize("T", [9, 70])
def test_partly_filled_row_tiles(kw, T):
    _check(configs.scaled(configs.NEMOTRON_Q4_0, E=4, top_k=2, **kw), T, prefill=True)


@pytest.mark.parametrize("types", [(formats.TYPE_Q5_K, formats.TYPE_Q5_K), (formats.TYPE_Q4_K, formats.TYPE_Q5_K), (formats.TYPE_Q5_K, formats.TYPE_Q6_K)], ids=str)
@pytest.mark.parametrize("H", [512, 1024, 3072])
@pytest.mark.parametrize("T", [8, 32, 33, 129])
def test_kquant_shared_expert_beside_packed_experts(types, H, T):
    _check(configs.scaled(IQ3, E=4, top_k=2, H=H, F=256, F_s=512, type_sh_gate_up=types[0], type_sh_down=types[1]), T, prefill=True)


# ... with the routed experts on the 16-pair tiles (up to five pairs per expert) and the K-quant tiles behind them, several of 32 tokens: the launches
# overlap, so the bits are looked at again and again
@pytest.mark.parametrize("types", [(formats.TYPE_Q5_K, formats.TYPE_Q5_K), (formats.TYPE_Q4_K, formats.TYPE_Q5_K)], ids=str)
@pytest.mark.parametrize("E,k,H", [(256, 8, 1024), (64, 2, 2048), (100, 3, 1024)])
@pytest.mark.parametrize("T", [33, 65, 129, 160])
def test_kquant_tiles_behind_tiles_of_sixteen_pairs(types, E, k, H, T):
    cfg = configs.scaled(IQ3, E=E, top_k=k, H=H, F=256, F_s=512, type_sh_gate_up=types[0], type_sh_down=types[1])
    _check(cfg, T, prefill=True)
    raw = configs.make_layer(cfg, device="cuda")
    tiled, pw, x = MoeWeightsTiled(raw), MoeWeightsPrefill(raw), configs.make_input(cfg, T, device="cuda")
    sc = MoeScratch(tiled, T)
    sc.enable_prefill()
    first = forward_moe_prefill(tiled, pw, sc, x)
    outs = [torch.empty_like(x) for _ in range(20)]
    for y in outs:
        forward_moe_prefill(tiled, pw, sc, x, y)
    assert all(torch.equal(y, first) for y in outs) and sc.status() == 0
    # Against the decode entry (K-quant GEMVs behind the routed part), also behind the residual and the norm: the same intermediates, the down rows' 16 sub-blocks
    # and the k + 1 rows of a token added in another order, i.e. at most 25 roundings of 2^-24 of sums up to twice the row's largest value: 3e-6
    # of that (3.3e-7 seen; one 8-bit step of an intermediate is 1e-4 and more).
    norm = torch.ones(H, device="cuda")
    half = [forward_moe_residual_norm(tiled, sc, x, torch.zeros_like(x), norm, 1e-6, None, p) for p in (pw, None)]
    for a, b in ((first, forward_moe(tiled, sc, x)), half):
        assert ((a - b).abs().amax(1) <= 3e-6 * b.abs().amax(1)).all()


# weights read packed and weights in operand order in one launch
@pytest.mark.parametrize("T", [20, 90])
def test_mixed_operand_forms(T):
    _check(configs.scaled(Q4, E=4, top_k=2, H=512, F=256, F_s=256, type_sh_gate_up=configs.Q8_0, type_sh_down=configs.Q8_0), T, prefill=True)


# ... enough wide tiles of both that every CTA goes from one form to the other, with more stages per tile than the rings have slots
def test_mixed_operand_forms_tile_after_tile():
    cfg = configs.scaled(Q4, E=4, top_k=2, H=2048, F=512, F_s=1024, type_sh_gate_up=configs.Q8_0, type_sh_down=configs.Q8_0)
    raw, T = configs.make_layer(cfg, device="cuda"), 2100
    tiled = MoeWeightsTiled(raw)
    x, sc = configs.make_input(cfg, T, device="cuda"), MoeScratch(tiled, T)
    want = forward_moe(tiled, sc, x).clone()      # (a Q8_0 shared expert keeps the decode entry on the GEMV kernels)
    pw = MoeWeightsPrefill(raw)
    for _ in range(5):
        check_rows(forward_moe_prefill(tiled, pw, sc, x).cpu().numpy(), want.cpu().numpy())
    assert sc.status() == 0


@pytest.mark.parametrize("cfg,T", [(configs.scaled(Q4, E=16, F=128, F_s=128, H=512), t) for t in (16, 17, 24, 25, 40, 41, 64)] +
                                  [(configs.scaled(configs.NEMOTRON_Q4_0, E=8, H=2688, F=800, F_s=1600, name="wide experts"), t) for t in (8, 16, 17, 33)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_decode_entry_steps(cfg, T):
    _check(cfg, T, prefill=False)


# rows of 1 .. 4 kilo-elements (one to four quads per partial), ragged ones, token counts around a tile of 32
@pytest.mark.parametrize("H", [256, 1024, 1152, 2048, 2688, 3200, 4096])
@pytest.mark.parametrize("T", [129, 160, 545])
def test_tiled_router(H, T):
    _check(configs.scaled(Q4, E=256, H=H, F=64, F_s=64), T, prefill=False)


# ... and around a tile of 16 and the line between the two, with a last tile of a few experts
@pytest.mark.parametrize("E,H,T", [(70, 4096, 239), (70, 3200, 465), (70, 1152, 471), (72, 2048, 944), (72, 2048, 945), (200, 1024, 335)])
def test_tiled_router_of_small_tiles(E, H, T):
    _check(configs.scaled(Q4, E=E, H=H, F=64, F_s=64), T, prefill=False)


# rows of up to one kilo-element on both sides of the tiled product's line, which counts the outputs for those of more than 512 columns
@pytest.mark.parametrize("E,H,T", [(128, 512, 289), (128, 512, 513), (128, 640, 288), (128, 640, 289), (36, 1024, 1024), (36, 1024, 1025)])
def test_tiled_router_of_short_rows(E, H, T):
    _check(configs.scaled(Q4, E=E, H=H, F=64, F_s=64), T, prefill=False)


# The decode entry runs pair by pair, on the 16-pair tiles or on the GEMM; a token's row is the same bits on each of them (the first two here,
# the GEMM in the next test), whatever the batch: odd numbers of K slices and units, IQ3_S in both places, a shared expert narrower than the routed ones.
@pytest.mark.parametrize("cfg", [configs.scaled(Q4, E=16, F=256, F_s=512, H=2048, name="q4"),
                                 configs.scaled(IQ3, E=16, F=512, F_s=256, H=1024, type_down=configs.IQ3_S, name="iq3"),
                                 configs.scaled(IQ3, E=8, top_k=4, F=320, F_s=0, H=2560, name="iq3 gate, q4 down"),
                                 configs.scaled(configs.NEMOTRON_Q4_0, E=8, H=2688, F=800, F_s=96, name="relu"),
                                 configs.scaled(IQ3, E=16, F=256, F_s=512, H=1024, type_sh_gate_up=formats.TYPE_Q5_K, type_sh_down=formats.TYPE_Q5_K, name="q5k")],
                         ids=lambda c: c.name)
@pytest.mark.parametrize("T", [17, 41, 64, 150])
def test_decode_rows_do_not_depend_on_the_batch(cfg, T):
    tiled = MoeWeightsTiled(configs.make_layer(cfg, device="cuda"))
    x = configs.make_input(cfg, T, device="cuda")
    sc, one = MoeScratch(tiled, T), MoeScratch(tiled, 1)
    y = forward_moe(tiled, sc, x)
    single = torch.cat([forward_moe(tiled, one, x[t:t + 1].contiguous()) for t in range(T)])
    assert sc.status() == 0 and one.status() == 0
    assert torch.equal(y, single)


# ... on the GEMM itself and the GEMV kernels behind it: experts and shared expert of different packed types, rows that the tiles' shared memory does
# not hold, and batches above the tiles' last one
@pytest.mark.parametrize("cfg,T", [(c, t) for c in (configs.scaled(IQ3, E=32, top_k=4, H=1024, F=256, F_s=256, type_sh_gate_up=configs.Q4_0, name="iq3, q4 shared"),
                                                    configs.scaled(Q4, E=32, top_k=4, H=1024, F=256, F_s=512, type_sh_gate_up=configs.IQ3_S, type_sh_down=configs.IQ3_S, name="q4, iq3 shared"),
                                                    configs.scaled(Q4, E=16, top_k=4, H=5120, F=128, F_s=128, name="rows of 5120"),
                                                    configs.scaled(configs.NEMOTRON_Q4_0, E=32, top_k=3, H=5120, F=800, F_s=96, name="relu, rows of 5120")) for t in (17, 41, 64, 150)] +
                                  [(configs.scaled(IQ3, E=16, H=4096, F=512, F_s=256, type_down=d, name="above the tiles"), 330) for d in (configs.Q4_0, configs.IQ3_S)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_decode_rows_on_the_gemm_do_not_depend_on_the_batch(cfg, T):
    raw = configs.make_layer(cfg, device="cuda")
    tiled, x = MoeWeightsTiled(raw), configs.make_input(cfg, T, device="cuda")
    sc, one = MoeScratch(tiled, T), MoeScratch(tiled, 1)
    y = forward_moe(tiled, sc, x)
    assert torch.equal(y, torch.cat([forward_moe(tiled, one, x[t:t + 1].contiguous()) for t in range(T)]))
    assert sc.status() == 0 and one.status() == 0
    if T <= 64:
        check_rows(y.cpu().numpy(), oracle_on_gpu_routing(raw.to("cpu"), x.cpu().numpy(), sc.topk_indices(T).cpu().numpy())["y"])


# a workspace for more tokens than the call has: the smaller batch may cut its pairs into more entries than the full one
@pytest.mark.parametrize("kw", [dict(E=8), dict(E=16), dict(E=64), dict(E=4, top_k=2, F_s=0)], ids=str)
@pytest.mark.parametrize("max_T", [25, 32, 40, 64])
def test_smaller_batches_in_a_larger_workspace(kw, max_T):
    cfg = configs.scaled(Q4, **{**dict(H=512, F=128, F_s=128), **kw})
    raw = configs.make_layer(cfg, device="cuda")
    tiled = MoeWeightsTiled(raw)
    sc = MoeScratch(tiled, max_T)
    for T in (24, 24, 8, 25, 24):
        x = configs.make_input(cfg, T, device="cuda")
        y = forward_moe(tiled, sc, x)
        torch.cuda.synchronize()
        assert sc.status() == 0
        idx = sc.topk_indices(T).cpu().numpy()
        check_rows(y.cpu().numpy(), oracle_on_gpu_routing(raw.to("cpu"), x.cpu().numpy(), idx)["y"])
        perm, offs = oracle.permute(idx, cfg.E)
        assert np.array_equal(sc.perm(T).cpu().numpy(), perm) and np.array_equal(sc.offsets().cpu().numpy(), offs)


# Eight tokens of one expert: an entry each where several CTAs share an SM, one entry for all where a CTA's weights fill it (Q8_0) and on
# raw blocks, which a kernel unpacks once per entry.
@pytest.mark.parametrize("cfg,packed,entries", [(Q4, True, 8), (IQ3, True, 8), (Q8, True, 1), (Q4, False, 1)], ids=lambda v: getattr(v, "name", str(v)))
def test_pairs_per_entry(cfg, packed, entries):
    raw = configs.make_layer(configs.scaled(cfg, E=1, top_k=1, H=512, F=256, F_s=0, zipf_bias=False), device="cuda")
    w = MoeWeightsTiled(raw) if packed else raw
    sc = MoeScratch(w, 64)
    route_only(w, sc, configs.make_input(configs.scaled(cfg, H=512), 8, device="cuda"))
    assert sc._view(sc.ws.group_list, 16).view(torch.int32).tolist() == [entries, entries, 0, 0]


# An output is a float pointer and may start on any float (a view into a larger buffer), also where the combine stores four at a time.
@pytest.mark.parametrize("T", [8, 64, 200])
@pytest.mark.parametrize("entry", ["decode", "host", "prefill"])
def test_outputs_on_any_float_boundary(entry, T):
    cfg = configs.scaled(Q4, E=16, F=128, F_s=128, H=512)
    raw = configs.make_layer(cfg, device="cuda")
    tiled = MoeWeightsTiled(raw)
    x, sc = configs.make_input(cfg, T, device="cuda"), MoeScratch(tiled, T)
    pw = MoeWeightsPrefill(raw)
    results = []
    for shift in range(4):
        room = torch.zeros(T * cfg.H + 4, pin_memory=entry == "host") if entry == "host" else torch.zeros(T * cfg.H + 4, device="cuda")
        y = room[shift:shift + T * cfg.H].reshape(T, cfg.H)
        if entry == "decode":
            forward_moe(tiled, sc, x, y)
        elif entry == "host":
            forward_moe_host(tiled, sc, x.cpu().pin_memory(), y)
        else:
            forward_moe_prefill(tiled, pw, sc, x, y)
        torch.cuda.synchronize()
        rest = room.cpu()
        assert sc.status() == 0 and rest[:shift].abs().sum() == 0 and rest[shift + T * cfg.H:].abs().sum() == 0
        results.append(y.cpu().clone())
    assert all(torch.equal(r, results[0]) for r in results)


# the taps of the intermediates after a decode call: the planes hold what the Q8_1 rows hold, for every pair and the shared expert
@pytest.mark.parametrize("cfg", [configs.scaled(IQ3, E=8, top_k=4, H=512, F=256, F_s=512), configs.scaled(configs.NEMOTRON_Q4_0, E=8, top_k=2, H=384, F=160, F_s=96)],
                         ids=lambda c: c.name)
@pytest.mark.parametrize("T", [8, 64])
def test_intermediates_as_planes(cfg, T):
    tiled = MoeWeightsTiled(configs.make_layer(cfg, device="cuda"))
    sc = MoeScratch(tiled, T)
    forward_moe(tiled, sc, configs.make_input(cfg, T, device="cuda"))
    pairs, wide = T * cfg.top_k, max(cfg.F, cfg.F_s)
    rows, stride = sc.inter_q8(T), (wide // 32 + 3) & ~3
    q = sc._view(sc.ws.inter_q, (pairs + T) * wide).reshape(pairs + T, wide)
    d = sc._view(sc.ws.inter_d, (pairs + T) * stride * 4).view(torch.float32).reshape(pairs + T, stride)
    for part, width in ((slice(0, pairs), cfg.F), (slice(pairs, pairs + T), cfg.F_s)):
        blocks = rows[part, :width // 32 * 36].reshape(-1, width // 32, 36)
        assert torch.equal(q[part, :width].reshape(-1, width // 32, 32), blocks[..., 4:])
        assert torch.equal(d[part, :width // 32], blocks[..., :2].contiguous().view(torch.float16)[..., 0].float())


# the prefill entry with fewer pairs than half the experts, and with one token more
@pytest.mark.parametrize("cfg", [configs.scaled(IQ3, E=32, H=512, F=256, F_s=256), configs.scaled(Q8, E=32, H=512, F=64, F_s=64),
                                 configs.scaled(IQ3, E=32, H=1024, F=256, F_s=512, type_sh_gate_up=formats.TYPE_Q5_K, type_sh_down=formats.TYPE_Q5_K, name="q5k")],
                         ids=lambda c: c.name)
@pytest.mark.parametrize("T", [1, 2, 3])
def test_prefill_entry_of_a_few_tokens(cfg, T):
    _check(cfg, T, prefill=True)


# one or two router rows per CTA: around one CTA per SM; a single row of inputs is always on pairs of router rows
@pytest.mark.parametrize("E,T", [(73, 9), (74, 9), (147, 8), (148, 8), (36, 32), (37, 32), (8, 1)])
@pytest.mark.parametrize("H", [2048, 2176])
def test_small_router(E, T, H):
    _check(configs.scaled(Q4, E=E, H=H, F=64, F_s=64), T, prefill=False)


# more token tiles than a grid's second dimension holds, on the simple router (one routed expert per token leaves the tiled one no scratch)
def test_router_of_many_tokens():
    cfg = configs.scaled(Q4, E=4, top_k=1, H=128, F=32, F_s=0)
    tiled, T, n = MoeWeightsTiled(configs.make_layer(cfg, device="cuda")), 8 * 65535 + 13, 64
    x = configs.make_input(cfg, T, device="cuda")
    sc, small = MoeScratch(tiled, T), MoeScratch(tiled, n)
    route_only(tiled, sc, x)
    ids = sc.topk_indices(T).flatten()
    assert sc.status() == 0
    for part in (slice(0, n), slice(T - n, T)):
        route_only(tiled, small, x[part].contiguous())
        assert torch.equal(sc.router_logits(T)[part], small.router_logits(n)) and torch.equal(ids[part], small.topk_indices(n).flatten())
    assert torch.equal(sc.perm(T).long(), torch.argsort(ids, stable=True))


# pairs as items of their own: rows of one unit to several K slices, slices and groups that are not full, more items than CTAs, warps that
# carry two slices, layers without a shared expert
@pytest.mark.parametrize("cfg", [configs.scaled(Q4, E=64, H=128, F=32, F_s=64, top_k=1), configs.scaled(Q4, E=64, H=1152, F=96, F_s=32, top_k=3),
                                 configs.scaled(IQ3, E=64, H=4096, F=256, F_s=256, top_k=8), configs.scaled(IQ3, E=64, H=256, F=512, F_s=0, type_down=configs.IQ3_S),
                                 configs.scaled(configs.NEMOTRON_Q4_0, E=64, H=2688, F=1856, F_s=3712, top_k=6),
                                 configs.scaled(configs.NEMOTRON_Q4_0, E=32, H=640, F=800, F_s=1600, top_k=2),
                                 configs.scaled(configs.NEMOTRON_Q4_0, E=32, H=384, F=1120, F_s=0, top_k=8)],
                         ids=lambda c: f"{c.name}-{c.H}-{c.F}-{c.F_s}-{c.top_k}")
@pytest.mark.parametrize("T", [1, 2, 5, 10, 40])
def test_pairs_as_items(cfg, T):
    _check(cfg, T, prefill=False)


# 16 pairs of an expert per tile: one column to a full tile and one more, eight and nine (the MMA's halves), ragged row tiles and K slices
@pytest.mark.parametrize("cfg", [configs.scaled(Q4, E=1, top_k=1, H=512, F=256, F_s=256), configs.scaled(IQ3, E=1, top_k=1, H=1280, F=256, F_s=0),
                                 configs.scaled(configs.NEMOTRON_Q4_0, E=1, top_k=1, H=640, F=1120, F_s=96), configs.scaled(Q4, E=3, top_k=2, H=128, F=64, F_s=64),
                                 configs.scaled(IQ3, E=5, top_k=4, H=2048, F=512, F_s=512, type_down=configs.IQ3_S)], ids=lambda c: f"{c.name}-{c.H}-{c.F}-{c.F_s}")
@pytest.mark.parametrize("T", [5, 8, 9, 15, 16, 17, 33, 70])
def test_tiles_of_sixteen_pairs(cfg, T):
    _check(cfg, T, prefill=False)


# ... and in the prefill entry, which takes them for small layers too: every token on the same experts, the batch the column count
@pytest.mark.parametrize("cfg", [configs.scaled(Q4, top_k=1, H=512, F=256, F_s=256), configs.scaled(IQ3, top_k=1, H=1280, F=256, F_s=0),
                                 configs.scaled(configs.NEMOTRON_Q4_0, top_k=1, H=640, F=1120, F_s=96), configs.scaled(Q4, top_k=2, H=128, F=64, F_s=64),
                                 configs.scaled(IQ3, top_k=4, H=2048, F=512, F_s=512, type_down=configs.IQ3_S)], ids=lambda c: f"{c.name}-{c.H}-{c.F}-{c.F_s}")
@pytest.mark.parametrize("T", [5, 8, 9, 15, 16, 17, 33, 70])
def test_tiles_of_sixteen_pairs_in_prefill(cfg, T):
    cfg = configs.scaled(cfg, E=max(cfg.top_k + 1, -(-T * cfg.top_k // 5)))   # (the fewest experts with which the batch is one for these tiles)
    raw = configs.make_layer(cfg, device="cuda")
    raw.router_bias = torch.zeros(cfg.E, device="cuda")
    raw.router_bias[:cfg.top_k] = 40.0
    tiled, x = MoeWeightsTiled(raw), configs.make_input(cfg, T, device="cuda")
    sc = MoeScratch(tiled, T)
    y = forward_moe_prefill(tiled, MoeWeightsPrefill(raw), sc, x)
    idx = sc.topk_indices(T).cpu().numpy()
    assert sc.status() == 0 and sc.offsets().cpu().tolist() == [min(i, cfg.top_k) * T for i in range(cfg.E + 1)]
    check_rows(y.cpu().numpy(), oracle_on_gpu_routing(raw.to("cpu"), x.cpu().numpy(), idx)["y"])
    assert torch.equal(y, forward_moe(tiled, sc, x))      # (the pairs' bits)


# small layers run pair by pair up to 64 tokens, on the work list up to 40 where a shared expert of one row tile makes the rows of a slice too
# long for the pair kernels
@pytest.mark.parametrize("cfg", [configs.scaled(Q4, E=8, top_k=2, H=256, F=64, F_s=64), configs.scaled(IQ3, E=64, H=512, F=256, F_s=0),
                                 configs.scaled(configs.NEMOTRON_Q4_0, E=1, top_k=1, H=384, F=96, F_s=96), configs.scaled(Q4, E=8, top_k=2, H=512, F=2880, F_s=32)],
                         ids=lambda c: f"{c.name}-{c.H}-{c.F}-{c.F_s}")
@pytest.mark.parametrize("T", [6, 33, 40, 41, 64, 65])
def test_small_layers_pair_by_pair(cfg, T):
    _check(cfg, T, prefill=False)
    tiled, x = MoeWeightsTiled(configs.make_layer(cfg, device="cuda")), configs.make_input(cfg, T, device="cuda")
    sc = MoeScratch(tiled, T)
    y = forward_moe(tiled, sc, x)
    assert torch.equal(torch.cat([forward_moe(tiled, sc, x[t:t + 1].contiguous()) for t in range(T)]), y) and sc.status() == 0


# a K-quant shared expert beside the pair kernels: one and two rows per step, every type, against the oracle and, bit for bit, against the
# launches of its own that a larger batch takes
@pytest.mark.parametrize("types", [(formats.TYPE_Q5_K, formats.TYPE_Q5_K), (formats.TYPE_Q4_K, formats.TYPE_Q6_K), (formats.TYPE_Q6_K, formats.TYPE_Q4_K)], ids=str)
@pytest.mark.parametrize("H,F_s", [(256, 256), (1024, 512), (2048, 768), (1280, 1024), (2304, 512)])
def test_kquant_shared_expert_beside_pairs(types, H, F_s):
    cfg = configs.scaled(IQ3, E=64, top_k=8, H=H, F=256, F_s=F_s, type_sh_gate_up=types[0], type_sh_down=types[1])
    raw = configs.make_layer(cfg, device="cuda")
    tiled, T = MoeWeightsTiled(raw), 48
    x, sc = configs.make_input(cfg, T, device="cuda"), MoeScratch(tiled, 48)
    y = forward_moe(tiled, sc, x)
    for n in (1, 4, 5, 10):
        part = torch.cat([forward_moe(tiled, sc, x[t:t + n].contiguous()) for t in range(0, 20, n)])
        assert torch.equal(part, y[:20]), n
    _check(cfg, 3, prefill=False)
    assert sc.status() == 0


# ... rows of two sub-blocks per lane, whose sums meet in a lane before they meet across the warp: enough tokens that a sum which is rounded
# differently shows in some intermediate's 8 bits
@pytest.mark.parametrize("type_gate_up", [formats.TYPE_Q4_K, formats.TYPE_Q5_K, formats.TYPE_Q6_K])
def test_kquant_rows_do_not_depend_on_the_batch(type_gate_up):
    cfg = configs.scaled(IQ3, E=32, top_k=2, H=2048, F=512, F_s=512, type_sh_gate_up=type_gate_up, type_sh_down=formats.TYPE_Q4_K)
    tiled, T = MoeWeightsTiled(configs.make_layer(cfg, device="cuda")), 400
    x, sc = configs.make_input(cfg, T, device="cuda"), MoeScratch(tiled, T)
    y = forward_moe(tiled, sc, x)
    for n in (5, 2):
        assert torch.equal(torch.cat([forward_moe(tiled, sc, x[t:t + n].contiguous()) for t in range(0, T, n)]), y), n
    assert sc.status() == 0


# residual + norm inside the router (up to four tokens, rows of up to 3072) and as a launch in front of it: the same bits, also in place
@pytest.mark.parametrize("H", [256, 2048, 2176, 3072, 3200])
@pytest.mark.parametrize("cfg", [Q4, configs.scaled(IQ3, type_sh_gate_up=formats.TYPE_Q5_K, type_sh_down=formats.TYPE_Q5_K)], ids=["q4", "q5k"])
def test_residual_norm_in_the_router(cfg, H):
    if H % 256 and cfg is not Q4:
        pytest.skip("IQ3_S rows are multiples of 256")
    cfg = configs.scaled(cfg, E=64, H=H, F=256, F_s=256)
    tiled = MoeWeightsTiled(configs.make_layer(cfg, device="cuda"))
    sc, gen = MoeScratch(tiled, 12), torch.Generator(device="cuda").manual_seed(H)
    hidden, residual = (torch.randn(12, H, generator=gen, device="cuda") for _ in range(2))
    norm = 1.0 + 0.1 * torch.randn(H, generator=gen, device="cuda")
    res = residual.clone()
    y = forward_moe_residual_norm(tiled, sc, hidden, res, norm, 1e-6)
    assert torch.equal(res, hidden + residual)
    for n in (1, 2, 3, 4):
        part = residual.clone()
        rows = [forward_moe_residual_norm(tiled, sc, hidden[t:t + n].contiguous(), part[t:t + n], norm, 1e-6) for t in range(0, 12, n)]
        assert torch.equal(torch.cat(rows), y) and torch.equal(part, res), n
    assert sc.status() == 0


# equal probabilities everywhere: the lowest indices win, in the kernels that select their experts themselves and at the router's end
@pytest.mark.parametrize("E,k", [(256, 8), (33, 8), (8, 8), (64, 1)])
@pytest.mark.parametrize("T", [1, 3, 40])
def test_equal_experts(E, k, T):
    cfg = configs.scaled(Q4, E=E, top_k=k, H=256, F=64, F_s=64)
    raw = configs.make_layer(cfg, device="cuda")
    raw.router_weight[:] = raw.router_weight[0]
    tiled = MoeWeightsTiled(raw)
    sc, x = MoeScratch(tiled, T), configs.make_input(cfg, T, device="cuda")
    forward_moe(tiled, sc, x)
    want = torch.arange(k, device="cuda", dtype=torch.int32).expand(T, k)
    assert torch.equal(sc.topk_indices(T), want)
    forward_moe(tiled, sc, torch.zeros_like(x))
    route_only(tiled, sc, x)
    assert torch.equal(sc.topk_indices(T), want) and sc.status() == 0


# rows from pinned memory (on any float boundary), from pageable memory, around the size up to which a kernel fetches them
@pytest.mark.parametrize("T", [1, 5, 32, 33])
def test_host_rows(T):
    cfg = configs.scaled(Q4, E=64, H=2048, F=64, F_s=64)
    tiled = MoeWeightsTiled(configs.make_layer(cfg, device="cuda"))
    sc, x = MoeScratch(tiled, T), configs.make_input(cfg, T, device="cuda")
    want = forward_moe(tiled, sc, x).cpu()
    for shift in (0, 1, 2, None):
        room = torch.empty(T * cfg.H + 4, pin_memory=shift is not None)
        rows = room[shift or 0:(shift or 0) + T * cfg.H].reshape(T, cfg.H)
        rows.copy_(x)
        y = torch.empty(T, cfg.H, pin_memory=True)
        for _ in range(3):   # (new values in the same buffer are seen)
            rows.neg_()
            forward_moe_host(tiled, sc, rows, y)
        assert torch.equal(y, forward_moe(tiled, sc, -x).cpu())
        rows.neg_()
        assert torch.equal(forward_moe_host(tiled, sc, rows, y), want)


# ... with a K-quant shared expert: inside the pair launches (up to five tokens) the result goes straight to pinned memory on any float boundary
@pytest.mark.parametrize("T", [1, 4, 5, 6])
def test_host_rows_kquant(T):
    cfg = configs.scaled(IQ3, E=64, H=1024, F=256, F_s=512, type_sh_gate_up=formats.TYPE_Q5_K, type_sh_down=formats.TYPE_Q5_K)
    tiled = MoeWeightsTiled(configs.make_layer(cfg, device="cuda"))
    sc, x = MoeScratch(tiled, T), configs.make_input(cfg, T, device="cuda")
    want = forward_moe(tiled, sc, x).cpu()
    for shift in (0, 1, 2, 3, None):
        room = torch.zeros(T * cfg.H + 4, pin_memory=shift is not None)
        at = shift or 0
        y = room[at:at + T * cfg.H].reshape(T, cfg.H)
        for rows in (x.cpu().pin_memory(), x.cpu()):
            y.zero_()
            assert torch.equal(forward_moe_host(tiled, sc, rows, y), want)
        assert room[:at].abs().sum() == 0 and room[at + T * cfg.H:].abs().sum() == 0
    assert sc.status() == 0


# rows that begin in pinned memory and end outside it are refused before a kernel touches them, on either side of the call
@pytest.mark.parametrize("T", [1, 4])
def test_host_rows_pinned_in_part(T):
    cfg = configs.scaled(Q4, E=16, H=2048, F=64, F_s=64)
    tiled = MoeWeightsTiled(configs.make_layer(cfg, device="cuda"))
    sc, x = MoeScratch(tiled, T), configs.make_input(cfg, T, device="cuda")
    want, cudart, page = forward_moe(tiled, sc, x).cpu(), torch.cuda.cudart(), 4096
    room = np.zeros(T * cfg.H + 3 * page // 4, np.float32)
    skip = -room.ctypes.data % page // 4
    rows = torch.from_numpy(room[skip:skip + T * cfg.H].reshape(T, cfg.H))   # (from a page's start)
    rows.copy_(x)
    for pages in (1, T * cfg.H * 4 // page):
        assert int(cudart.cudaHostRegister(rows.data_ptr(), pages * page, 0)) == 0
        y, x_pinned = torch.empty(T, cfg.H).pin_memory(), x.cpu().pin_memory()
        if pages == 1:
            for a, b in ((rows, y), (x_pinned, rows)):
                with pytest.raises(RuntimeError, match="-101"):
                    forward_moe_host(tiled, sc, a, b)
        else:
            assert torch.equal(forward_moe_host(tiled, sc, rows, y), want) and torch.equal(forward_moe_host(tiled, sc, x_pinned, rows), want)
        assert int(cudart.cudaHostUnregister(rows.data_ptr())) == 0
    assert sc.status() == 0


# the dispatch of a large batch: counts by the top-k kernel (four experts per token and more) and by a launch, chunks that 128 is no multiple
# of, a last chunk of one token, more chunks than a lane of the scan takes at a time
@pytest.mark.parametrize("k,T", [(1, 4096), (1, 4225), (3, 1366), (4, 1024), (6, 683), (7, 10009), (8, 512), (8, 513), (8, 8209)])
def test_dispatch_of_large_batches(k, T):
    cfg = configs.scaled(Q4, E=40, top_k=k, H=2048, F=32, F_s=0)
    tiled, x = MoeWeightsTiled(configs.make_layer(cfg, device="cuda")), configs.make_input(cfg, T, device="cuda")
    sc = MoeScratch(tiled, T)
    for _ in range(2):   # (the scratch is left as it was found)
        route_only(tiled, sc, x)
        ids = sc.topk_indices(T).flatten()
        assert torch.equal(sc.perm(T).long(), torch.argsort(ids, stable=True))
        assert torch.equal(sc.offsets().long(), torch.cat([ids.new_zeros(1), torch.bincount(ids, minlength=cfg.E).cumsum(0)]).long())
    assert sc.status() == 0


# ... numbers of chunks around a multiple of four, the most that one CTA scans and one more
@pytest.mark.parametrize("k,T", [(8, 528), (8, 529), (8, 545), (8, 576), (8, 1024), (8, 1025), (1, 4097), (6, 1324)])
def test_dispatch_of_few_chunks(k, T):
    test_dispatch_of_large_batches(k, T)


# Q8_1 of whole rows: rows of any float alignment, blocks of zeros, of tiny and huge values, of NaN and infinities, against the one-warp form
def test_rows_quantised_four_elements_per_lane():
    cfg = configs.scaled(Q4, E=128, top_k=1, H=1152, F=32, F_s=0)
    tiled, T = MoeWeightsTiled(configs.make_layer(cfg, device="cuda")), 600
    sc, small = MoeScratch(tiled, T), MoeScratch(tiled, 8)
    room = torch.empty(T * cfg.H + 1, device="cuda")
    for shift in (0, 1):
        x = room[shift:shift + T * cfg.H].reshape(T, cfg.H)
        x.copy_(configs.make_input(cfg, T, device="cuda"))
        x[0] = 0.0
        x[1] *= 1e-30
        x[2] *= 1e30
        x[3, 40], x[3, 70], x[3, 200] = float("nan"), float("inf"), -float("inf")
        x[4, ::3] = 0.0
        x[5, 32:64] *= 1e-38
        route_only(tiled, sc, x)
        route_only(tiled, small, x[:8].contiguous())
        assert torch.equal(sc.x_q8(T)[:8], small.x_q8(8))
