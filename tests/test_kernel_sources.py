"""What the kernels' sources promise and no single launch shows."""
import ctypes
import os
import re

import llm_infer_rust_b200.kernels.build as build


def test_launch_limits_do_not_follow_the_launches():
    """A kernel's limit of shared memory is set once, to one size.  Kept in a number that grows with the launches it could be set
    by two threads in the wrong order, the smaller size last and the larger one remembered; launches in between then fail."""
    seen = 0
    for name in sorted(os.listdir(build.CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(build.CSRC, name)) as f:
                text = f.read()
            seen += len(re.findall(r"\bstatic bool configured\b", text))
            grows = re.findall(r"\bstatic (?:size_t|int|unsigned|long long) configured\b.*", text)
            assert not grows, f"{name}: {grows}"
    assert seen > 5


def test_results_that_are_no_int_are_not_asked_for_through_the_binding():
    """The binding calls every entry point as one that returns an int; a wider result has to come through the library itself."""
    wide = set()
    for name in sorted(os.listdir(build.CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(build.CSRC, name)) as f:
                wide.update(re.findall(r"^B200_EXPORT (?!int )[\w ]+?[ *](b200_\w+)\(", f.read(), re.M))
    assert len(wide) > 3
    package, asked = os.path.dirname(build.CSRC), 0
    for folder, _, files in os.walk(package):
        for name in (n for n in files if n.endswith(".py")):
            with open(os.path.join(folder, name)) as f:
                lines = f.read().splitlines()
            for i, line in enumerate(lines):
                for receiver, entry in re.findall(r"((?:\w|\.|\(\))+)\.(b200_\w+)\b(?=\()", line):
                    if entry in wide:
                        asked += 1
                        itself = receiver.endswith(".library") or any(f"{receiver} = load_cuda_library(" in p for p in lines[max(0, i - 5):i])
                        assert itself, f"{name}:{i + 1}: {line.strip()}"
    assert asked > 2


def test_blocks_that_share_a_tile_of_32_bit_products():
    """Measured with every count of blocks (148 SMs): the fullest SM's time decides, two blocks on an SM cost as much as one."""
    lib = build.load_cuda_library("gemm_f32.cu")

    def shared(m, n, k):
        tiles, spans = -(-m // 64) * -(-n // 64), -(-k // 512)
        return lib.b200_gemm_f32_blocks_a_tile(ctypes.c_longlong(tiles), spans, 148)
    for m, n, k, blocks in ((64, 4096, 1024, 2), (128, 4096, 1024, 2), (48, 6144, 1024, 2), (500, 1024, 2048, 4), (500, 1024, 3072, 6),
                            (128, 4096, 2048, 4), (64, 4096, 4096, 8), (300, 24576, 4096, 8), (64, 4096, 12288, 8), (17, 64, 300, 1)):
        assert shared(m, n, k) == blocks, (m, n, k)
    # nine or ten spans take two rounds with five blocks or with eight: the three more would only add a round to nothing
    assert shared(64, 64, 5000) == 5 and shared(64, 64, 4500) == 5 and shared(64, 64, 4096) == 8


def test_heads_that_a_lane_group_takes_between_projection_and_attention():
    """A decode step's few tokens take the shortest chain, a prompt's many the fewest fetches (measured on both sides)."""
    lib = build.load_cuda_library("qkv_post.cu")
    taken = lambda tokens, heads, lanes: lib.b200_qkv_post_heads_a_group(ctypes.c_longlong(tokens * heads), lanes)
    assert [taken(t, 32, 16) for t in (1, 27, 64, 200, 300, 500, 777, 8192)] == [1, 1, 1, 1, 2, 2, 4, 4]       # bfloat16, heads of 128
    assert [taken(t, 32, 32) for t in (4, 64, 128, 200, 300, 2048)] == [1, 1, 2, 2, 4, 4]                      # float32


def test_gates_take_eight_elements_a_thread_where_that_is_faster():
    lib = build.load_cuda_library("gated.cu")
    eight = lambda tokens, width: bool(lib.b200_sigmoid_gate_mul_takes_eight(tokens, width))
    assert not any(eight(t, w) for t, w in ((1, 8), (300, 256), (300, 768), (64, 512), (1500, 512)))
    assert all(eight(t, w) for t, w in ((1, 2048), (300, 1024), (1500, 768), (8192, 512)))


def test_columns_that_a_warp_takes_of_few_rows_experts():
    """Two while the grid fills the SMs and experts have few rows each (measured on both sides)."""
    cols = build.load_cuda_library("experts.cu").b200_experts_few_cols
    assert cols(1024, 8, 64) == cols(2048, 64, 64) == cols(1536, 8, 8) == cols(2048, 2, 8) == 2
    assert cols(256, 4, 4) == cols(512, 32, 4) == 1                         # 64 and 128 blocks
    assert cols(1536, 64, 8) == cols(768, 32, 8) == 1                       # four and eight rows an expert


def test_many_tokens_walk_between_projection_and_attention():
    """bfloat16 from more than six blocks an SM on (measured on both sides), float32 never."""
    walks = build.load_cuda_library("qkv_post.cu").b200_qkv_post_walks
    threads = lambda tokens, heads: ctypes.c_longlong(tokens * (heads // 2) * 16)
    assert all(walks(1, threads(t, h)) for t, h in ((1020, 32), (2048, 48), (8192, 32)))
    assert not any(walks(1, threads(t, h)) for t, h in ((777, 32), (500, 32), (45, 48))) and not walks(0, threads(8192, 32))


def test_up_to_four_rows_of_32_bit_products():
    """Which of the two kernels for few rows, by what each costs over the SMs (measured on both sides, 148 SMs)."""
    groups = lambda m, n, k: build.load_cuda_library("gemm_f32.cu").b200_gemm_f32_pair_groups(m, n, k, 148)
    assert all(groups(m, n, k) == 1 for m in (1, 4) for n, k in ((1024, 2048), (1024, 3072), (256, 1024)))
    assert all(groups(m, n, k) == 2 for m in (1, 2) for n, k in ((151936, 1024), (24576, 4096), (6144, 4096), (16384, 1536)))
    assert groups(1, 4096, 12288) == 2 and groups(2, 2048, 8192) == groups(4, 2048, 4096) == 1
    assert not any(groups(m, n, k) for m, n, k in ((1, 4096, 1024), (1, 16384, 512), (4, 4096, 512), (4, 24576, 4096), (2, 16384, 8192), (4, 6144, 4096), (5, 1024, 3072)))


def test_which_kernel_takes_a_32_bit_product_in_terms():
    """By rows and by what each costs over the SMs (measured on both sides, 148 SMs)."""
    route = build.load_cuda_library("gemm_f32.cu").b200_gemm_f32_route
    few = lambda m, n, k: route(m, n, k, 148) == 0
    assert all(few(m, n, k) for m in (1, 8, 16) for n, k in ((1024, 3072), (151936, 1024), (24576, 4096)))
    assert few(48, 2048, 2048) and few(64, 2048, 2048)          # (clusters of eight would take two rounds)
    assert few(32, 4096, 1024) and few(32, 6144, 1024) and few(64, 1024, 2048) and few(64, 1024, 3072) and few(96, 1024, 2048) and few(128, 64, 1024)
    assert not any(few(m, n, k) for m, n, k in ((32, 151936, 1024), (64, 4096, 4096), (64, 24576, 4096), (128, 6144, 1024), (129, 64, 64), (300, 1024, 2048)))
