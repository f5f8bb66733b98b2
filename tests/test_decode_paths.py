"""Host-side logic of the decode-sized kernels' wrappers: CPU fallbacks equal the plain formulas and the path predicates
refuse what the kernels do not take (the kernels themselves are tested on a GPU in test_gpu_kernels.py / test_moe.py /
test_qwen35.py)."""
import pytest
import torch

from tyr_b200.models.common import KVCache
from tyr_b200.ops import decode_attention as DA
from tyr_b200.ops import decode_gemm as DG
from tyr_b200.ops import delta_rule as DR
from tyr_b200.ops import fp4
from tyr_b200.ops import prompt_mix as PM
from tyr_b200.ops import rope as RO
from tyr_b200.ops import skinny as SK
from tyr_b200.ops.gemm import gemm, gemm_many


def test_decode_gemm_cpu_fallback_and_predicate():
    g = torch.Generator().manual_seed(0)
    x = torch.randn(20, 128, generator=g).bfloat16()
    wg = (torch.randn(256, 128, generator=g) * 0.1).bfloat16()
    wu = (torch.randn(256, 128, generator=g) * 0.1).bfloat16()
    assert not DG.supported(x, wg) and not DG.supported(x, wg, wu, min_tiles=1)       # CPU tensors never take the kernel
    ref = x.float() @ wg.float().T
    assert torch.equal(DG.decode_linear(x, wg), ref.to(torch.bfloat16))
    out = torch.zeros(20, 256 + 8, dtype=torch.bfloat16)
    DG.decode_linear(x, wg, out=out[:, 8:])
    assert torch.equal(out[:, 8:], ref.to(torch.bfloat16)) and torch.equal(out[:, :8], torch.zeros(20, 8, dtype=torch.bfloat16))
    gated = (torch.nn.functional.silu(ref) * (x.float() @ wu.float().T)).to(torch.bfloat16)
    assert torch.equal(DG.decode_swiglu(x, wg, wu), gated)


def test_decode_gemm_thresholds_are_ordered():
    # the gated form is taken from fewer tiles than the plain one, and the plain one has an upper bound
    assert DG.MIN_ROWS == 17 and DG.MAX_ROWS == 64
    assert 1 <= DG.MIN_ROW_TILES <= DG.MAX_ROW_TILES
    assert DG.GATED_MIN_ROW_TILES >= 1


def test_fixed_slot_predicate():
    assert not fp4.fixed_slots_supported(129, 2048)            # an expert could receive more rows than a slot tile holds
    assert not fp4.fixed_slots_supported(64, 2048 + 64)        # hidden size must be a multiple of 256
    assert fp4.FIXED_SLOT_MAX_TOKENS == 128
    assert fp4.scatter_fits(256) and fp4.scatter_fits(21760) and not fp4.scatter_fits(22016)      # four rows of codes and scales in 48 KB
    assert not fp4.fixed_slots_supported(64, 22016)


def test_gdr_tile_predicate_needs_aligned_rows(monkeypatch):
    monkeypatch.setattr(DR, "_GDR_TILE_MIN_TILES", 0)
    v = torch.zeros(4, 1, 8 * 128, dtype=torch.bfloat16)
    assert not DR._tile_ok(64, v, None, 32)                     # value head width other than 128
    z = torch.zeros(4, 1, 8 * 128 + 2, dtype=torch.bfloat16)[..., :8 * 128]
    if DR._tile_ok(128, v, None, 32):                            # only when the library carries the kernel
        assert not DR._tile_ok(128, v, z, 32)                    # row stride not a multiple of 4 elements
        monkeypatch.setattr(DR, "_GDR_TILE_MIN_TILES", 64)
        assert not DR._tile_ok(128, v, None, 32)                 # fewer tiles than the threshold


def test_slices_fill_the_chip_without_a_thin_last_wave():
    """The fastest (or next to it) of the measured numbers of slices, for few and many pairs, short and long stores."""
    for (B, G, keys, heads, D), good in {(1, 2, 564, 4, 256): {9}, (32, 4, 576, 4, 256): {2}, (40, 4, 2048, 4, 256): {3}, (72, 4, 8192, 4, 256): {1},
                                         (32, 4, 2048, 4, 128): {3}, (38, 4, 8192, 4, 128): {2, 5, 6}, (48, 4, 8192, 4, 128): {2}, (64, 4, 2048, 4, 128): {3},
                                         (40, 4, 2048, 8, 64): {4}, (38, 4, 8192, 8, 64): {4}, (75, 4, 8192, 8, 64): {2},
                                         (16, 4, 200, 8, 256): {1}, (8, 4, 129, 8, 256): {1}, (8, 4, 1000, 16, 64): {4, 5, 6, 8, 10}}.items():
        assert DA.pick_splits(B, G, keys, heads, D, D) in good, (B, G, keys, D)
    for keys in (1, 64, 65, 300, 100000):
        for B in (1, 7, 150, 100000):
            assert 1 <= DA.pick_splits(B, 2, keys) <= min(32, -(-keys // 64))


def test_prompt_operands_refuse_what_the_kernel_would_read_beyond():
    B, S, H, G, D, half = 2, 5, 4, 2, 64, 16
    bf = lambda *s: torch.zeros(s, dtype=torch.bfloat16)
    q, k, v, w, tab = bf(B, S, H * 2 * D), bf(B, S, G * D), bf(B, S, G * D), bf(D), torch.zeros(S, half)
    store = KVCache.allocate(B, G, S, D, "cpu", torch.bfloat16)
    assert PM.operands_fit(q, k, v, store, w, w, tab, D, tab)
    one = torch.zeros(1, half)                                     # a single position's turn broadcast over the prompt
    for bad in ((q, k, v, store, w, w, one, D, one), (q, k, v, store, w, w, tab, D, one), (q, k, v, store, w[:1], w, tab, D, tab),
                (q, k[..., :D], v, store, w, w, tab, D, tab), (q, k, v[..., :D], store, w, w, tab, D, tab), (q[..., :H * D + D], k, v, store, w, w, tab, D, tab),
                (q, k, v, KVCache.allocate(B, G + 1, S, D, "cpu", torch.bfloat16), w, w, tab, D, tab), (q, k[:1], v, store, w, w, tab, D, tab)):
        assert not PM.operands_fit(*bad)
    for heads, tables in (((H + 1, G), tab), ((H, G + 1), tab), ((H, G), one)):
        with pytest.raises(ValueError, match="heads of"):
            PM.attention_operands(q, 2 * D, k, v, w, w, tables, tables, 1e-6, *heads, D, store)
    assert store.length == 0


def test_delta_gates_leave_other_types_and_strides_to_the_plain_operations():
    wide, p = torch.zeros(2, 7, 24, dtype=torch.bfloat16), torch.zeros(8)
    b, a = wide[..., :8], wide[..., 8:16]
    assert DR.gates_fit(b, a, p, p) and DR.gates_fit(b.float(), a.float(), p, p) and DR.gates_fit(b[:, :1], a[:, :1], p, p)
    for t in (torch.float16, torch.float64):
        assert not DR.gates_fit(b.to(t), a.to(t), p, p)
    assert not DR.gates_fit(b, a.float(), p, p) and not DR.gates_fit(b, a, p.half(), p) and not DR.gates_fit(b, a, p, torch.zeros(16)[::2])
    assert not DR.gates_fit(b[:, :5], a[:, :5], p, p) and not DR.gates_fit(b.mT.contiguous().mT, a.mT.contiguous().mT, p, p)
    assert not DR.gates_fit(b, a, p[:1], p) and not DR.gates_fit(b, a, p, p.reshape(1, 8))


def test_product_forms_refuse_operands_of_other_types_and_devices():
    bf = lambda *s: torch.ones(s, dtype=torch.bfloat16)
    a, w, aux, gate = bf(6, 16), bf(8, 16), bf(6, 8), bf(2, 8)
    assert gemm(a, w, up=w, act="swiglu").shape == gemm(a, w, act="gated_add", aux=aux, gate=gate).shape == (6, 8)
    for t in (torch.float32, torch.int8, torch.float16):
        with pytest.raises(TypeError, match="up"):
            gemm(a, w, up=w.to(t), act="swiglu")
    there = torch.device("meta")
    for kw in (dict(up=w.to(there), act="swiglu"), dict(act="gated_add", aux=aux, gate=gate.to(there))):
        with pytest.raises(ValueError, match="meta"):
            gemm(a, w, **kw)
    for short in (aux[:5], aux[:, :4], aux[None]):
        with pytest.raises(ValueError, match="gated_add"):
            gemm(a, w, act="gated_add", aux=short, gate=gate)
    with pytest.raises(ValueError, match="meta"):
        gemm_many(a, [w, w.to(there)])


def test_norm_products_refuse_operands_that_do_not_go_together():
    bf = lambda *s: torch.ones(s, dtype=torch.bfloat16)
    x, n, w = bf(3, 64), bf(64), bf(16, 64)
    assert SK.norm_fit(x, None, n, [w]) and SK.norm_fit(x, x, n, [w, w])
    for bad in ((x, x.float(), n, [w]), (x, x[:2], n, [w]), (x, x, n.float(), [w]), (x, x, n[:32], [w]), (x, x, n, [w, w.float()]), (x, x, n, [w[:, :32]]),
                (x, x, n, [w.to("meta")])):
        assert not SK.norm_fit(*bad)
    with pytest.raises(ValueError, match="bf16 operands"):
        SK.skinny_norm_many(x, x.float(), n, 1e-6, [w])
    with pytest.raises(ValueError, match="differ"):
        SK.skinny_norm_swiglu(x, x, n, 1e-6, w, w[:8])


def test_turned_queries_and_keys_go_together():
    bf, tab, pos = lambda *s: torch.ones(s, dtype=torch.bfloat16), torch.ones(9, 8), torch.zeros(3, dtype=torch.int32)
    q, k, w = bf(3, 4, 32), bf(3, 2, 32), bf(32)
    assert RO.qk_fit(q, k, tab, tab, w, w, pos)
    for bad in ((q, k[:2], tab, tab, w, w, pos), (q, bf(3, 2, 16), tab, tab, w, w, pos), (q, k, tab, tab[:4], w, w, pos), (q, k, tab, tab, w[:1], w, pos),
                (q, k, tab, tab, w, w, pos[:1]), (q, k, tab, tab, w, w.float(), pos), (q, k, tab, tab, w, w, pos.to("meta"))):
        assert not RO.qk_fit(*bad)


def test_matrices_share_a_launch_where_that_is_the_faster_way():
    for M, K, widths, want in ((1, 5120, (12288, 1024, 1024), [1, 2]), (8, 4096, (1024, 12288, 1024), [0, 2]), (9, 5120, (12288, 1024, 1024), [0, 1, 2]),
                               (1, 1024, (6144, 2048, 16, 16), [0, 1, 2, 3]), (4, 5120, (10240, 6144, 48, 48), [0, 1, 2, 3]), (1, 4096, (16384, 1024, 1024), [0, 1, 2]),
                               (20, 5120, (4096,), []), (32, 4096, (2048, 2048), []), (20, 5120, (48, 48), [0, 1]), (32, 5120, (1024, 1024), [0, 1]),
                               (20, 1024, (4096, 512, 512), [0, 1, 2]), (32, 8192, (3072, 64), [1]), (16, 64, (7,), [0]), (3, 64, (), [])):
        assert SK.shared_launch(M, K, widths) == want, (M, K, widths)
