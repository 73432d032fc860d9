"""Which kernel a step's work goes to: decisions taken on the host from sizes alone (no GPU, nothing launched)."""
import torch

from jllm_serve_b200.csrc import ops


def test_product_kernel_by_rows_and_shape():
    k = ops.gemm_kernel_for
    assert k(1, 4096, 4096) == "rows"
    assert k(8, 24576, 4096) == "rows"                     # few rows: even the widest matrix goes row by row
    assert k(16, 24576, 4096) == "tiles"                   # 16 rows against gate_up: tcgen05 tiles
    assert k(16, 6144, 4096) == "rows"
    assert k(17, 6144, 4096) == "swap"                     # QKV (50 MB) from 17 rows: weight rows as the MMA's M side
    assert k(64, 6144, 4096) == "swap" and k(128, 6144, 4096) == "swap" and k(129, 6144, 4096) == "tiles"
    assert k(161, 6144, 4096) == "tiles" and k(161, 4096, 4096) == "tiles"      # above 128 rows its parked parts cost too much
    # ... except against matrices much longer than high (down), up to the 256 tokens of one tcgen05 N side
    assert k(64, 4096, 12288) == "swap" and k(128, 4096, 12288) == "swap" and k(212, 4096, 12288) == "swap" and k(257, 4096, 12288) == "tiles"
    assert k(256, 5120, 17408) == "swap" and k(200, 24576, 4096) == "tiles"
    assert k(513, 4096, 12288) == "tiles" and k(400, 6144, 4096) == "tiles" and k(400, 4096, 12288, pairs=0) == "tiles"
    assert k(40, 4096, 4096) == "rows" and k(41, 4096, 4096) == "swap"         # O (34 MB): from 41 rows
    assert k(64, 24576, 4096) == "tiles"                                       # gate_up: whole tiles fill the SMs
    # many rows: two SMs to a 256 x 256 tile where such tiles keep the pairs busy in no more rounds than one-SM tiles
    assert k(2048, 4096, 4096) == "pair" and k(2048, 6144, 4096) == "pair" and k(2048, 24576, 4096) == "pair"
    assert k(1024, 4096, 12288) == "pair" and k(512, 24576, 4096) == "pair"
    assert k(512, 6144, 4096) == "tiles"                   # 48 tiles for 74 pairs
    assert k(300, 24576, 4096) == "tiles"                  # 300 rows: three 128-row tiles, not two of 256
    assert k(1024, 6144, 4096) == "tiles"                  # the one-SM kernel would take 192-wide tiles: 2 rounds of 0.83
    assert k(544, 5120, 5120) == "tiles" and k(544, 5120, 17408) == "tiles"     # a third pair tile an eighth full
    assert k(2048, 4096, 4096, pairs=0) == "tiles"         # a device that runs no pairs
    assert k(16, 24576, 4096, tiles_fit=False) == "rows"
    assert k(8, 4096, 4096, rows_fit=False) == "tiles"
    assert k(8, 4096, 4096, rows_fit=False, tiles_fit=False) == ""


def test_decode_attention_splits_fill_the_gpu_once():
    scratch = torch.empty(2 << 20)
    # 8 rows x 8 kv heads = 64 pairs for 296 places: 4 blocks per pair; 16 keys-of-256 allow up to 32
    assert ops.decode_splits(8, 8, 16, 32, 128, scratch, places=296) == 4
    assert ops.decode_splits(1, 8, 16, 32, 128, scratch, places=296) == 32      # one row: as many as the keys allow, 32 at most
    assert ops.decode_splits(1, 8, 2, 32, 128, scratch, places=296) == 4        # 512 keys: blocks of at least 128
    assert ops.decode_splits(64, 8, 16, 32, 128, scratch, places=296) == 1
    assert ops.decode_splits(8, 8, 16, 32, 128, None, places=296) == 1          # no scratch, no partial results
    tiny = torch.empty(8 * 32 * 2 * (128 + 2))                      # room for two splits only
    assert ops.decode_splits(8, 8, 16, 32, 128, tiny, places=296) == 2


def test_decode_attention_is_dealt_out_evenly_only_where_that_pays():
    scratch = torch.empty(2 << 20)
    assert ops.decode_plan(8, 8, 16, 32, 128, scratch, places=296) == ("split", 4)          # fewer pairs than places
    assert ops.decode_plan(37, 8, 16, 32, 128, scratch, places=296) == ("split", 1)         # 296 pairs: one full round
    how, blocks = ops.decode_plan(64, 8, 16, 32, 128, scratch, places=296)                  # 512 pairs: 1.73 rounds
    assert how == "flat" and blocks == 296
    how, blocks = ops.decode_plan(104, 3, 1, 6, 64, scratch, places=296)                    # few kv heads bound the blocks
    assert how == "flat" and blocks == 62 * 3
    assert ops.decode_plan(64, 8, 16, 32, 80, scratch, places=296)[0] == "split"            # a head size the flat kernel lacks
    assert ops.decode_plan(64, 8, 16, 32, 128, torch.empty(1000), places=296)[0] == "split"  # no room for its partial results


def test_a_decode_steps_bucket_is_clamped_where_it_stops_mattering():
    """`decode_bucket_cap`: from that bucket on the plan of a decode step is the same for every longer context, so the
    step function may clamp the bucket there (and a growing context does not ask for a new captured step every 256
    tokens); below it the bucket is rounded down to one of sixteen levels, each a valid plan for fewer keys."""
    import torch
    from jllm_serve_b200.csrc import ops
    scratch = torch.empty(2 << 20)
    for rows, heads, kv_heads, hd, window in [(1, 32, 8, 128, 0), (8, 32, 8, 128, 0), (64, 32, 8, 128, 0), (3, 40, 8, 128, 0),
                                              (8, 64, 8, 128, 0), (200, 6, 3, 64, 0), (2, 16, 1, 256, 0), (8, 32, 8, 128, 700),
                                              (1, 4, 4, 64, 5000), (37, 8, 2, 64, 0)]:
        cap = ops.decode_bucket_cap(rows, kv_heads, heads, hd, window, scratch, places=296)
        assert 1 <= cap <= ops.KV_BUCKET_MAX

        def plan(b):
            return ops.decode_plan(rows, kv_heads, ops._windowed_bucket(b, window), heads, hd, scratch, 296)
        for b in range(1, ops.KV_BUCKET_MAX + 1):
            assert plan(min(b, cap)) == plan(b), (rows, heads, kv_heads, hd, window, b, cap)
        assert cap == 1 or plan(cap - 1) != plan(cap)
    assert ops.decode_bucket_cap(8, 8, 32, 128, 0, scratch, places=296) == 2       # four splits from 512 keys on
    assert ops.decode_bucket_cap(1, 8, 32, 128, 0, scratch, places=296) == 16      # 32 splits from 4,096 keys on
    levels = [ops.bucket_level(b) for b in range(0, 40)]
    assert levels[:9] == [1, 1, 2, 3, 4, 5, 6, 7, 8] and levels[32:] == [32] * 8
    assert all(l <= max(1, b) and l in ops.KV_BUCKET_LEVELS for b, l in enumerate(levels))
    assert all(4 * b <= 5 * l + 4 for b, l in enumerate(levels[:33]))                # never more than a quarter below
    assert len(set(levels)) == 16


def test_what_the_recurrence_chunks_take_is_asked_once_per_shape(monkeypatch):
    """Launches and workspace of a step's chunks: one launch and nothing where the segments are short, three for a long one, four where
    both are there; passes over the heads where a pass's states fill 256 MB. A second layer of the step asks nothing."""
    ops._chunk_plan.cache_clear()
    plan = lambda *shape: ops._chunk_plan(*shape)
    assert plan(64, 1, 64, 64, 8, 128, 64) == (0, 1) and plan(33, 33, 1, 64, 8, 128, 64) == (0, 1)
    floats, launches = plan(2048, 1, 2048, 64, 8, 128, 64)
    assert launches == 3 and floats == 33 * 64 * (128 * 64 + 1)
    assert plan(2080, 33, 2048, 64, 8, 128, 64)[1] == 4                   # 32 single rows beside a portion
    assert plan(1100, 1, 1100, 256, 256, 128, 128)[1] == 6 and plan(1100, 1, 1100, 256, 256, 128, 128)[0] <= 64 << 20
    floats, launches = plan(2048, 8, 256, 64, 8, 128, 64)                 # eight of 256: their blocks fill the SMs
    assert (floats, launches) == (0, 1)
    monkeypatch.setattr(ops, "library", lambda: (_ for _ in ()).throw(AssertionError("the library was asked again")))
    assert plan(64, 1, 64, 64, 8, 128, 64) == (0, 1)
    ops._chunk_plan.cache_clear()


def test_a_wait_that_ran_out_is_reported_with_its_kernel(monkeypatch):
    """Every code that a kernel's source raises in an error word is named as that kernel's, and the report says so."""
    import re
    from pathlib import Path

    import pytest
    folder, seen = Path(ops.__file__).parent, 0
    for file in sorted(list(folder.glob("*.cu")) + list(folder.glob("*.cuh"))):
        text = file.read_text()
        codes = [int(c) for c in re.findall(r"atomicExch\((?:a\.)?error_word, (?:warp == 4 \? )?(\d+)", text) + re.findall(r"give_up\((\d+)\)", text)
                 + re.findall(r"warp == 4 \? \d+ : (\d+)\)", text)]
        for code in codes:
            word = "products" if file.stem.startswith("gemm") else "attention"
            assert ops.wait_kernel(word, code).split()[0] == file.stem, (file.name, code)
        seen += len(codes)
    assert seen >= 25

    class Fake:
        def __init__(self, products, attention):
            self.jllm_gemm_tcgen05_error, self.jllm_attention_prefill_tc_error = lambda: products, lambda: attention
            self.jllm_checks_bounds = lambda: 0
    for products, attention, what in ((16, 0, r"inside gemm_stream \(clusters\) \(code 16\)$"), (0, 51, r"inside attention_decode_ring \(code 51\)$"),
                                      (2, 43, r"gemm_tcgen05 \(code 2\), attention_prefill_latent \(code 43\)$")):
        monkeypatch.setattr(ops, "library", lambda: Fake(products, attention))
        with pytest.raises(ops.KernelError, match=what):
            ops.check_kernel_errors()
    monkeypatch.setattr(ops, "library", lambda: Fake(0, 0))
    ops.check_kernel_errors()


def test_products_of_129_to_256_rows_are_counted_on_both_kernels():
    """`gemm_stream` cuts k up over all SMs, the tiles walk all of it: what is long for its rows goes there, what is short or has enough
    tiles does not (each shape was measured on both)."""
    k = ops.gemm_kernel_for
    for rows, n, kk in ((144, 512, 16384), (256, 512, 16384), (240, 1024, 8192), (256, 2048, 12288), (256, 1536, 8960), (200, 2048, 8192),
                        (160, 4096, 8192), (212, 4096, 12288), (144, 256, 4096), (144, 5120, 5120), (212, 5120, 17408), (150, 2048, 5120)):
        assert k(rows, n, kk) == "swap", (rows, n, kk)
    for rows, n, kk in ((130, 4096, 4096), (160, 6144, 4096), (144, 7168, 5120), (144, 2048, 2048), (150, 4096, 512), (150, 512, 128),
                        (256, 768, 3072), (256, 2048, 5120), (256, 4096, 8192), (150, 1024, 2816), (240, 256, 4096)):
        assert k(rows, n, kk) == "tiles", (rows, n, kk)
    assert k(200, 4096, 12288, tiles_fit=False) == "" and k(256, 2048, 5120, sms=1000) == "swap"


def test_a_product_asks_once_which_kernel_takes_it(monkeypatch):
    """Alignment, SMs and pairs are asked once a product, the choice is worked out once per size: prompts of some hundreds of rows wait
    for the host, and a product's choice is a part of its launch."""
    asked = []

    def counted(name, answer):
        monkeypatch.setattr(ops, name, lambda *a, **k: (asked.append(name), answer(*a, **k))[1])
    counted("_tcgen05_fits", ops._tcgen05_fits)
    counted("sm_count", lambda: 148)
    counted("resident_pairs", lambda: 74)
    counted("gemm_kernel_for", ops.gemm_kernel_for)
    for name in ("gemm_small_m", "gemm_stream", "gemm_tcgen05", "gemm_pair"):
        monkeypatch.setattr(ops, name, lambda *a, name=name, **k: asked.append(name))
    ops.product_choice.cache_clear()
    for rows, n, k, kernel in ((8, 4096, 4096, "gemm_small_m"), (64, 6144, 4096, "gemm_stream"), (613, 4096, 4096, "gemm_tcgen05"),
                               (2048, 24576, 4096, "gemm_pair"), (300, 3072, 512, "gemm_tcgen05")):
        w = ops.PackedWeight(torch.zeros(1, dtype=torch.bfloat16).expand(-(-n // 128), -(-k // 64), 1), n, k)
        a, out = torch.zeros(rows, k, dtype=torch.bfloat16), torch.zeros(1)
        asked.clear()
        ops.gemm_bf16(a, w, out)
        ops.gemm_bf16(a, w, out)
        assert asked.count(kernel) == 2 and asked.count("gemm_kernel_for") == 1, asked
        assert asked.count("_tcgen05_fits") == 2 and asked.count("sm_count") == 2 and asked.count("resident_pairs") == (2 if rows > 128 else 0), asked
    assert ops.product_choice(64, 4096, 4096, fits=False) == ""
    ops.product_choice.cache_clear()


def test_the_kernel_bench_names_the_kernel_that_runs(monkeypatch):
    """`kernel_bench`'s label of a product is the kernel that `gemm_bf16` calls, and that kernel is one of those it times side by side."""
    from jllm_serve_b200.kernel_bench import product_kernels
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    monkeypatch.setattr(ops, "resident_pairs", lambda: 74)
    ran = []
    for name in ("gemm_small_m", "gemm_stream", "gemm_tcgen05", "gemm_pair"):
        monkeypatch.setattr(ops, name, lambda a, w, out, *args, name=name, **more: ran.append((name, args, more)))
    seen = set()
    for rows in (8, 47, 64, 150, 200, 300, 613, 1024, 2048):
        for n, k in ((6144, 4096), (4096, 4096), (24576, 4096), (4096, 12288)):
            chosen, kernels = product_kernels(ops, rows, n, k, 74 if rows > 128 else 0)
            w = ops.PackedWeight(torch.zeros(1, dtype=torch.bfloat16).expand(-(-n // 128), -(-k // 64), 1), n, k)
            ran.clear()
            ops.gemm_bf16(torch.zeros(1, dtype=torch.bfloat16).expand(rows, k).contiguous(), w, torch.zeros(1))
            fn, more = kernels[chosen]
            by_bench = ran.pop()
            fn(None, None, None, **more)
            assert ran[-1][0] == by_bench[0], (rows, n, k, chosen)
            seen.add(chosen)
    assert seen == {"rows", "swap", "tiles", "pair"}
