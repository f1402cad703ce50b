"""How many CTAs share a row's keys in decode attention (``parts/attention.py::decode_splits``): the rule's decisions
at the shapes that the measurements behind it used (148 SMs)."""
from llm_infer_rust_b200.parts.attention import decode_splits


def test_a_grid_that_fills_the_sms_stays_whole():
    # 32 and 64 rows x 8 KV heads: whole, although two or four splits would fill the last wave better
    # (measured: 90.8 against 103.8 us, 177.5 against 182.3 us at 4,096 keys a row)
    for ctas in (130, 256, 512, 4096):
        for keys in (512, 4096, 65536):
            assert decode_splits(ctas, keys, 148) == 1


def test_small_grids_are_split_to_fill_the_sms():
    assert decode_splits(64, 4096, 148) == 2          # 8 rows x 8 KV heads: 128 CTAs, a cluster of two combines them
    assert decode_splits(32, 4096, 148) == 4
    assert decode_splits(8, 4096, 148) == 8           # one row: eight clusters of eight
    assert decode_splits(16, 4096, 148) == 7          # two rows: eight would be sixteen clusters of eight, which do not find room
    # every CTA keeps at least 512 keys
    assert decode_splits(8, 512, 148) == 1 and decode_splits(8, 1024, 148) == 2
    assert decode_splits(0, 4096, 148) == decode_splits(1, 4096, 148)


def test_a_bound_beyond_the_rows_does_not_leave_the_wave():
    # 8 rows x 8 KV heads in a graph for up to 8,192 or 40,960 keys: two splits (one wave, one cluster), not the nine that
    # fill four waves best (576 CTAs on 148 SMs; measured: 38 against 47 us at 4,096 keys a row)
    for bound in (4096, 8192, 40960):
        assert decode_splits(64, bound, 148) == 2 and decode_splits(32, bound, 148) == 4 and decode_splits(96, bound, 148) == 1
    # one row: a cluster of eight until rows may be long, then as many as fill the wave
    assert decode_splits(8, 8192, 148) == 8 and decode_splits(8, 40960, 148) == 18
    for ctas in range(1, 200):
        for bound in (1, 511, 512, 4096, 131072):
            s = decode_splits(ctas, bound, 148)
            assert s == 1 or (s * ctas <= 148 and s * 512 <= bound)


def test_the_benchmark_asks_for_the_splits_that_the_engine_takes():
    """Latent rows (one KV head, values in the key rows) have a rule of their own: 8 rows x 16 heads of 320 columns, 2,048 keys,
    sixteen splits; one row sixteen too.  The benchmark times the kernels it names with what the engine's parts ask for."""
    import pathlib
    import torch
    from llm_infer_rust_b200.parts import attention as parts
    latent = lambda rows, bound=2048: parts.attention_splits(torch.bfloat16, rows, 16, 1, 320, 16, bound, 148, 256, True)
    assert latent(1) == latent(8) == 16 and latent(16) == 9
    # a wave filled with six or three splits, not clusters of four or two (24 rows: 21.7 against 37 us, with 32 heads 77 against 141)
    assert latent(24) == 6 and parts.attention_splits(torch.bfloat16, 24, 32, 1, 448, 16, 2048, 148, 384, True) == 3
    grouped = lambda rows, bound, dtype=torch.bfloat16: parts.attention_splits(dtype, rows, 16, 8, 128, 16, bound, 148)
    assert grouped(8, 4096) == 2 and grouped(1, 4096) == 8 and grouped(64, 4096) == 1
    assert grouped(4, 900, torch.float32) == 4           # the all-sizes kernel is split from 128 keys on
    bench = (pathlib.Path(parts.__file__).parents[2] / "bench.py").read_text()
    assert "decode_splits" not in bench and bench.count("attention_splits(") >= 6


def test_long_rows_on_few_sms_are_split_beyond_clusters_and_waves():
    """At the shapes that were measured (16 query and 8 KV heads of 128): what is faster at a quarter of the bound and beyond, never
    a count that short bounds would pay for."""
    import torch
    from llm_infer_rust_b200.parts.attention import attention_splits
    splits = lambda rows, bound: attention_splits(torch.bfloat16, rows, 16, 8, 128, 16, bound, 148)
    assert splits(3, 8192) == 4 and splits(3, 40960) == 6
    assert splits(5, 4096) == 2 and splits(5, 8192) == splits(5, 40960) == 3          # two left 68 of 148 SMs idle
    assert splits(6, 4096) == 2 and splits(6, 40960) == 3
    assert splits(10, 8192) == 1 and splits(10, 12288) == 3 and splits(10, 40960) == 5          # whole left 68 idle
    assert splits(12, 8192) == 1 and splits(12, 40960) == 3
    for rows in (4, 7, 8, 9, 14, 15, 16, 17, 19, 32, 64):                             # nothing is to be had, or whole waves as they are
        assert splits(rows, 40960) == (4 if rows == 4 else 2 if rows < 10 else 1)
    for rows in range(1, 70):
        for bound in (1, 300, 1024):
            assert splits(rows, bound) <= max(1, bound // 512)
        for bound in (4096, 8192, 40960, 131072):
            assert 1 <= splits(rows, bound) <= 64 and splits(rows, bound) * rows * 8 <= max(4 * 148, rows * 8)


def test_small_heads_of_the_all_sizes_kernel_fill_every_cta_that_an_sm_holds():
    """Float32 heads of 32: three CTAs an SM (measured at 4,096 keys: 8 and 16 rows x 8 KV heads 32.5 and 55 us in six and three splits, whole
    115 and 118); heads of 128 leave room for one."""
    import torch
    from llm_infer_rust_b200.kernels import ops
    from llm_infer_rust_b200.parts.attention import attention_splits
    assert ops.all_sizes_decode_ctas_per_sm(torch.float32, 32) == 3 and ops.all_sizes_decode_ctas_per_sm(torch.float32, 128) == 1
    splits = lambda rows, nh, nkv, d, bound=4096: attention_splits(torch.float32, rows, nh, nkv, d, 16, bound, 148)
    assert [splits(r, 16, 8, 32) for r in (1, 4, 8, 16, 32)] == [8, 8, 6, 3, 1]
    assert splits(8, 40, 1, 32) == 5 and splits(4, 40, 1, 32) == 8 and splits(8, 16, 8, 32, 300) == 2
    assert [splits(r, 16, 8, 128) for r in (1, 4, 8, 16)] == [8, 4, 2, 1]
