"""Forms of the integer step's kernels for few rows and for prompts whose scores fit tensor memory, at the sizes where their branches meet."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import attention as oattn
from oracle import fixed_point as ofp
from tests.attn_util import device_pool
from tests.test_gpu_attention import _extend_case, eq, run_extend
from tests.test_gpu_pending import _layer, _linear_case, _workspaces_zero

pytestmark = pytest.mark.gpu


def d(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# One to eight CTAs per row, a last CTA or warp without a block, blocks up to the kernel's limit; values that need the saturating butterflies
@pytest.mark.parametrize("rows,inter", [(1, 128), (1, 1152), (3, 6400), (17, 12288), (64, 25600), (65, 3072), (37, 17 * 128), (2, 32768), (2, 49152)])
@pytest.mark.parametrize("block", [0, 128])
@pytest.mark.parametrize("top", [2**18, 2**22, 2**31 - 1])
def test_silu_of_few_rows(rows, inter, block, top):
    from mini_sgl_integer_b200.kernel import fixed_point as fp
    rng = np.random.default_rng(rows + inter)
    gu = rng.integers(-top, top, (rows, 2 * inter)).astype(np.int32)
    gu[0, :128] = 0
    act = ofp.silu_and_mul(gu)
    codes, scale, absmax = ofp.per_token_quant_from_q15(ofp.blockwise_fwht_q15(act, block) if block else act)
    got = fp.silu_mul_fwht_quant(d(gu), block)
    np.testing.assert_array_equal(got[0].cpu().numpy(), codes)
    np.testing.assert_array_equal(got[1].cpu().numpy().reshape(-1), np.asarray(scale).reshape(-1))
    np.testing.assert_array_equal(got[2].cpu().numpy().reshape(-1), np.asarray(absmax).reshape(-1))


# whole blocks only; a split tail inside the up half and across both; everything split; pairs of CTAs (more than 64 rows)
@pytest.mark.parametrize("m,inter,k", [(1, 128, 256), (3, 6400, 2048), (1, 12288, 1024), (37, 148 * 64, 512), (64, 3072, 1024), (65, 12288, 1024), (200, 9472 + 128, 512),
                                       (256, 1536, 2048)])
@pytest.mark.parametrize("shift", [True, False])
def test_activation_on_a_linear_with_a_pending_tail(m, inter, k, shift):
    from mini_sgl_integer_b200.kernel import fixed_point as fp
    from mini_sgl_integer_b200.layers.w8a8_int8 import W8A8Int8LinearMethod
    codes, absmax, w8, wm, ws, acc, q15 = _linear_case(m + inter + k, m, 2 * inter, k, shift)
    want = ofp.per_token_quant_from_q15(ofp.blockwise_fwht_q15(ofp.silu_and_mul(q15), 128))
    layer, method = _layer(w8, wm, ws), W8A8Int8LinearMethod()
    for _ in range(2):
        tail = method.apply_tail(layer, d(codes), d(absmax))
        np.testing.assert_array_equal(tail.out[:, :tail.tail_col0].cpu().numpy(), q15[:, :tail.tail_col0])
        got = fp.silu_mul_fwht_quant(tail, 128)
        np.testing.assert_array_equal(got[0].cpu().numpy(), want[0])
        np.testing.assert_array_equal(got[2].cpu().numpy().reshape(-1), want[2].reshape(-1))
        assert _workspaces_zero()


# One short of, at and beyond the 512 keys whose scores are kept, with and without a prefix; tiles of 64, 32, 16 and 8 tokens
@pytest.mark.parametrize("kv_heads", [1, 2, 4, 8])
@pytest.mark.parametrize("kv_len,q_len", [(511, 511), (512, 40), (513, 513), (640, 9), (577, 300), (64, 64), (65, 1)])
def test_tiled_prefill_around_the_kept_scores(kv_heads, kv_len, q_len):
    kv_lens, q_lens = [kv_len, 30], [q_len, 30]
    case = _extend_case(kv_len + q_len, kv_lens, q_lens, 8, kv_heads, 64)
    want = oattn.paged_attention(case["q8"], case["qm"], case["qs"], case["pool"], case["tables"], kv_lens, q_lens)
    eq(run_extend(case, device_pool(case, 64, kv_heads), 640, impl="tiled").cpu().numpy(), want)


@pytest.mark.parametrize("requests", [1, 5, 70])
def test_a_step_that_reads_ahead_gives_the_bits_of_one_that_does_not(requests):
    """Weights, gains, page tables and the keys of earlier steps are read before the wait on the kernels in front only inside a model's
    forward; the layers by themselves wait first."""
    from mini_sgl_integer_b200.attention import Int8PagedKVCache
    from mini_sgl_integer_b200.layers.decoder_layer import AttnBatch
    from mini_sgl_integer_b200.models import Qwen3ForCausalLMInteger, Qwen3IntegerConfig, random_weights
    cfg = Qwen3IntegerConfig(3, 512, 8, 2, 1536, 1000, max_pos=256)
    weights = random_weights(cfg, 5, generate_on_device=True)
    g = torch.Generator(device="cuda").manual_seed(7)
    lens = torch.randint(1, 120, (requests,), device="cuda", generator=g, dtype=torch.int32)
    table = torch.arange(requests * 8, dtype=torch.int32, device="cuda").view(requests, 8)
    loc = (table.gather(1, (lens - 1)[:, None].long() // 16)[:, 0] * 16 + (lens - 1) % 16).to(torch.int32)
    ids = torch.randint(0, 1000, (requests,), device="cuda", generator=g, dtype=torch.int32)
    batch = AttnBatch(lens - 1, loc, table, lens, None, 128)
    out = []
    for ahead in (True, False):
        pool = Int8PagedKVCache(2, 3, 128, requests * 8, "cuda")
        for i in range(3):
            gi = torch.Generator(device="cuda").manual_seed(i)
            for c in (pool.k_cache(i), pool.v_cache(i)):
                c.copy_(torch.randint(-127, 128, c.shape, dtype=torch.int8, device="cuda", generator=gi))
            meta = pool.meta(i)
            meta[:, :, :32] = 2**30 + 12345
            meta[:, :, 32:40] = 0x24242424
        model = Qwen3ForCausalLMInteger(cfg, weights, pool)
        if ahead:
            logits = model.forward(ids, batch)
        else:
            codes, absmax = model.model.forward(ids, batch)
            logits = model.method.apply_quantised(model.lm_head, codes, absmax)
        out.append([logits] + [t.clone() for i in range(3) for t in (pool.k_cache(i), pool.v_cache(i), pool.meta(i))])
    assert all(torch.equal(a, b) for a, b in zip(*out)) and _workspaces_zero()


# One more row than a decode batch, one to four parts of K, several token tiles, single CTAs (a short K), and too many tiles to be left pending
@pytest.mark.parametrize("m,n,k,pays", [(257, 2048, 512, True), (333, 4096, 4096, True), (333, 6144, 4096, True), (700, 3072, 2048, True), (1025, 1024, 4096, True),
                                        (2000, 128, 1024, True), (300, 1028, 128, True), (600, 8192, 512, False)])
def test_prompts_of_few_tiles_are_left_pending(m, n, k, pays):
    from mini_sgl_integer_b200.kernel import fixed_point as fp
    from mini_sgl_integer_b200.kernel.pending import leaves_pending
    from mini_sgl_integer_b200.layers.w8a8_int8 import W8A8Int8LinearMethod
    codes, absmax, w8, wm, ws, acc, q15 = _linear_case(m + n, m, n, k)
    assert leaves_pending(m, n) == pays
    layer, method = _layer(w8, wm, ws), W8A8Int8LinearMethod()
    rng = np.random.default_rng(m)
    res, gain = rng.integers(-(2**18), 2**18, (m, n)).astype(np.int32), rng.integers(2**13, 2**15, n).astype(np.int32)
    want, want_res = ofp.fused_add_rmsnorm_v2(res, q15, gain)
    for _ in range(2):
        pending = method.apply_pending(layer, d(codes), d(absmax))
        np.testing.assert_array_equal(pending.acc.cpu().numpy(), acc)
        got = fp.fused_add_rmsnorm_quant(pending, d(res), d(gain))
        np.testing.assert_array_equal(got[0].cpu().numpy(), ofp.per_token_quant_from_q15(want)[0])
        np.testing.assert_array_equal(got[3].cpu().numpy(), want_res)
        assert _workspaces_zero()


# One to 256 decoding requests (pending linears, the activation's tail), prompts of few tiles and of many; no shifts, no q/k norms
@pytest.mark.parametrize("lens,decode", [([40], True), ([5, 64, 33] * 9, True), ([17] * 200, True), ([3], False), ([100, 1, 60], False), ([300, 90], False), ([900, 1200], False)])
@pytest.mark.parametrize("plain", [True, False])
def test_layers_from_native_code_give_the_bits_of_their_own_forward(lens, decode, plain, monkeypatch):
    from mini_sgl_integer_b200 import _lib
    from mini_sgl_integer_b200.attention import Int8PagedKVCache
    from mini_sgl_integer_b200.layers.decoder_layer import AttnBatch
    from mini_sgl_integer_b200.models import Qwen3ForCausalLMInteger, Qwen3IntegerConfig, qwen3_integer, random_weights
    cfg = Qwen3IntegerConfig(3, 2304, 8, 2, 1280, 1000, max_pos=2048)
    weights = random_weights(cfg, 5, generate_on_device=True, qk_norm=plain)
    if not plain:
        weights["layers"][1]["gate_up"].weight_shift = weights["layers"][2]["o"].weight_shift = None
    g = torch.Generator(device="cuda").manual_seed(7)
    n, pitch = len(lens), -(-max(lens) // 16)
    table = torch.randperm(n * pitch, device="cuda", generator=g).to(torch.int32).view(n, pitch)
    kv = torch.tensor(lens, dtype=torch.int32, device="cuda")
    seq = torch.arange(n, device="cuda") if decode else torch.repeat_interleave(torch.arange(n, device="cuda"), kv.long())
    pos = kv.long() - 1 if decode else torch.cat([torch.arange(k, device="cuda") for k in lens])
    loc = (table[seq, pos // 16] * 16 + pos % 16).to(torch.int32)
    ids = torch.randint(0, 1000, (len(pos),), device="cuda", generator=g, dtype=torch.int32)
    batch = AttnBatch(pos.to(torch.int32), loc, table, kv, None if decode else kv, max(lens))
    out, calls = [], []
    for native in (True, False):
        pool = Int8PagedKVCache(2, 3, 128, n * pitch, "cuda")
        for i in range(3):
            gi = torch.Generator(device="cuda").manual_seed(i)
            for c in (pool.k_cache(i), pool.v_cache(i)):
                c.copy_(torch.randint(-127, 128, c.shape, dtype=torch.int8, device="cuda", generator=gi))
            meta = pool.meta(i)
            meta[:, :, :32], meta[:, :, 32:40] = 2**30 + 12345, 0x24242424
        model = Qwen3ForCausalLMInteger(cfg, weights, pool)
        run = qwen3_integer.run_layers
        took = []
        monkeypatch.setattr(qwen3_integer, "run_layers", (lambda *a: took.append(run(*a)) or took[-1]) if native else (lambda *a: None))
        before = _lib.CALLS
        logits = model.forward(ids, batch)
        calls.append(_lib.CALLS - before)
        monkeypatch.setattr(qwen3_integer, "run_layers", run)
        assert not native or took[0] is not None
        out.append([logits] + [t.clone() for i in range(3) for t in (pool.k_cache(i), pool.v_cache(i), pool.meta(i))])
    assert all(torch.equal(a, b) for a, b in zip(*out)) and _workspaces_zero() and calls[0] == calls[1]


# Eight lanes a row (more than 12284 rows of q, k and v heads) against a warp a row: head counts that leave warps partly empty, 8-byte constants, one norm,
# rows of zeros, of every magnitude up to the saturating ones and of -2^31, dropped places
@pytest.mark.parametrize("tokens,hq,hk", [(3072, 2, 1), (1759, 5, 1), (1367, 7, 1), (1400, 32, 8)])
@pytest.mark.parametrize("norms,fwht,shift", [("qk", True, 0), ("q", True, 2), ("", True, 2), ("k", False, 0)])
def test_qkv_rows_of_eight_lanes_have_the_bits_of_rows_of_a_warp(tokens, hq, hk, norms, fwht, shift):
    from mini_sgl_integer_b200.attention import Int8PagedKVCache, qkv_rope_quant_store
    g = torch.Generator(device="cuda").manual_seed(tokens + hq)
    ints = lambda lo, hi, *shape: torch.randint(lo, hi, shape, dtype=torch.int32, device="cuda", generator=g)
    heads, pages = hq + 2 * hk, tokens // 16 + 2
    x = ints(-2**31, 2**31 - 1, tokens, heads, 128) >> ints(0, 32, tokens, heads, 1)       # a magnitude per row: warps of small and of large rows, too
    x[::3] >>= 13
    x[5, 0], x[6, :], x[7, -1, 9], x[8, hq, 3] = 0, 0, -2**31, -2**31
    x = x.reshape(tokens, heads * 128)
    at = lambda t: torch.cat([t.new_zeros(shift), t.reshape(-1)])[shift:].view(t.shape)      # 8 bytes past a 16-byte boundary
    angle = torch.rand((300, 64), device="cuda", generator=g) * 6.3
    cache = at(torch.cat([angle.cos(), angle.sin()], 1).mul(32768).round().to(torch.int32))
    cache[17, 3] = 40000                                                                     # not of a rotation: the general form
    gains = {n: at(ints(2**11, 2**14, 128)) if n in norms else None for n in "qk"}
    pos, loc = ints(0, 300, tokens), torch.randperm(pages * 16, device="cuda", generator=g)[:tokens].to(torch.int32)
    loc[3], loc[4] = -1, pages * 16 + 5
    pool = [Int8PagedKVCache(hk, 1, 128, pages, "cuda") for _ in range(2)]
    for c in pool:
        c.k_cache(0).zero_(), c.v_cache(0).zero_(), c.meta(0).zero_()
    step = 12284 // heads
    run = lambda i, rows, src: qkv_rope_quant_store(pos[rows], src, hq, pool[i], 0, loc[rows], cache, gains["q"], gains["k"], with_fwht=fwht)
    parts = [run(0, slice(a, a + step), x[a:a + step]) for a in range(0, tokens, step)]
    want = [torch.cat(p) for p in zip(*parts)]
    got = run(1, slice(0, tokens), x)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert all(torch.equal(a, b) for f in ("k_cache", "v_cache", "meta") for a, b in [(getattr(pool[0], f)(0), getattr(pool[1], f)(0))])
