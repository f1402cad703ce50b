"""Kernels and branches at the sizes where their split of the work changes, against the same operation in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rnd(*shape, dtype=torch.float32, seed=0, scale=1.0):
    return (scale * torch.randn(*shape, generator=torch.Generator().manual_seed(seed))).to(DEV, dtype)


# rows at the edge of the two kernels (16, 17), one column beyond a tile, K around chunks (128), spans (512), more spans than
# warps (8), more than one span a block, odd K (no 16-byte loads), three passes over many columns (tiles) and two (streamed)
@pytest.mark.parametrize("m,n,k", [(1, 9, 127), (3, 8, 129), (16, 7, 513), (2, 24, 4500), (17, 65, 4100), (64, 64, 512), (65, 129, 1028),
                                   (300, 1024, 2048), (33, 130, 515), (16, 40, 9001), (5, 3000, 1024), (16, 1030, 3072), (9, 4100, 4500), (8, 4100, 4500)])
def test_32_bit_products(m, n, k):
    from llm_infer_rust_b200.kernels import ops
    a, w = _rnd(m, k), _rnd(n, k, seed=1)
    got = ops.gemm_f32(a, w)
    want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    # a chain of 128 sums, then 3, then K / 512: at most (131 + K / 512) roundings of 2^-24 of the terms' size
    assert ((got.double() - want).abs() <= (131 + k / 512) * 2.0 ** -24 * size).all()
    for r in {0, m // 2, m - 1}:                              # bit for bit what the row gives alone (the kernel for few rows)
        assert torch.equal(ops.gemm_f32(a[r:r + 1].contiguous(), w)[0], got[r])


# groups of 8, 16 and 32 rows of x and tiles of 64 and 128, each with a rest; one row of W beyond a tile; K of one stage (32), of spans of
# one stage and of several, with a rest; one, three, four and eight blocks a tile; few columns and many
@pytest.mark.parametrize("m,n,k", [(1, 127, 4), (9, 129, 32), (16, 2500, 36), (17, 128, 36), (32, 1024, 3072), (33, 257, 256), (64, 300, 260),
                                   (40, 20000, 1056), (65, 1024, 2048), (100, 30000, 256), (128, 130, 1056), (129, 640, 96), (257, 128, 8000),
                                   (300, 2500, 1024), (300, 1030, 3072), (4, 20000, 1024), (8, 4100, 12288)])
def test_32_bit_products_in_three_terms(m, n, k):
    from llm_infer_rust_b200.kernels import ops
    for offset in (0.0, 1.0):                                   # sums that cancel, and sums that grow
        a, w = _rnd(m, k) + offset, _rnd(n, k, seed=1) + offset
        got = ops.gemm_f32(a, w)
        want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
        # 32 k: twelve sums on the tensor cores, which may cut off a last place (2^-23) each; then K / 256 + 2 stages a span and
        # eight spans, roundings of 2^-24; what three of the nine products leave out is 2^-24 at most
        assert ((got.double() - want).abs() <= (24 + 1 + k / 256 + 10) * 2.0 ** -24 * size).all()
        # bit for bit what rows give alone and in the other kernels' counts
        for rows in (slice(0, 1), slice(m // 2, m // 2 + 1), slice(m - 1, m), slice(0, 8), slice(0, 16), slice(0, 50), slice(0, 130)):
            assert torch.equal(ops.gemm_f32(a[rows].contiguous(), w), got[rows])
        ops.check_errors(a.device)


@pytest.mark.parametrize("spread", [3.0, 8.0, None])
def test_32_bit_products_of_few_and_many_rows_have_the_same_bits(spread):
    """mma.sync and tcgen05 cut off what does not fit their sums at the same place, whatever the numbers: wide spreads, cancelling pairs."""
    from llm_infer_rust_b200.kernels import ops
    a, w = _rnd(140, 512), _rnd(20000, 512, seed=1)
    if spread is not None:
        a, w = a * torch.exp(spread * _rnd(140, 512, seed=2)), w * torch.exp(spread * _rnd(20000, 512, seed=3))
    else:
        a[:, 1::2], w[:, 1::2] = a[:, 0::2], -w[:, 0::2] * (1 + 1e-6 * _rnd(20000, 256, seed=4))
    whole = ops.gemm_f32(a, w)
    for rows in (8, 16, 32):
        assert torch.equal(torch.cat([ops.gemm_f32(a[i:i + rows].contiguous(), w) for i in range(0, 140, rows)]), whole)


def test_32_bit_products_of_infinities_and_the_largest_numbers():
    """A value without three finite terms: an infinity, a NaN, a number that rounds to a bfloat16 infinity."""
    from llm_infer_rust_b200.kernels import ops
    for m, n, k in ((3, 200, 256), (40, 130, 2048), (200, 300, 1024), (150, 20000, 64)):
        a, w = _rnd(m, k), _rnd(n, k, seed=1)
        a[0, 5], a[1, 9], a[2, 1], w[11, 4], w[5, 5] = float("inf"), float("nan"), 3.4e38, float("-inf"), 0.0
        w[:, 1] *= 0.1
        got, want = ops.gemm_f32(a, w), a.double() @ w.double().t()
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
        assert torch.equal(got[got.isinf()].double(), want[want.isinf()])
        fine = want.isfinite()
        assert fine[2].any() and ((got.double() - want).abs()[fine] <= 1e-5 * want.abs().clamp_min(10.0)[fine]).all()
    small, w = _rnd(5, 64) * 1e-30, _rnd(130, 64, seed=1)
    want, size = small.double() @ w.double().t(), small.double().abs() @ w.double().abs().t()
    assert ((ops.gemm_f32(small, w).double() - want).abs() <= 40 * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("exponent", [-105, -118, -126])
@pytest.mark.parametrize("m,n,k", [(5, 130, 64), (200, 300, 1024), (150, 20000, 64)])
def test_32_bit_products_of_very_small_numbers(m, n, k, exponent):
    """Above and below 2^-110, where a third term no longer has all its bits."""
    from llm_infer_rust_b200.kernels import ops
    for of_w in (False, True):
        a, w = _rnd(m, k).abs() + 1.0, _rnd(n, k, seed=1)
        a, w = (a, w * 2.0 ** exponent) if of_w else (a * 2.0 ** exponent, w)
        got = ops.gemm_f32(a, w)
        want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
        # as test_32_bit_products_in_three_terms, or k / 32 + 5 roundings of FFMA, and half of the smallest float32 for each of k + 40 sums
        assert ((got.double() - want).abs() <= (35 + k / 32) * 2.0 ** -24 * size + (k + 40) * 2.0 ** -150).all()
        assert torch.equal(ops.gemm_f32(a[2:5].contiguous(), w), got[2:5])


# up to four rows: one group of warps and two, tiles of eight rows of W with a rest, one tile, several a group, fewer than groups; K of odd
# counts of stages, of one stage more than eight spans, with a rest of a stage; spans that are empty; x that fits beside one ring only
@pytest.mark.parametrize("m,n,k,groups", [(1, 256, 1024, 1), (4, 1021, 1028, 1), (2, 9, 4100, 1), (3, 1184, 1060, 1), (1, 1185, 1024, 2), (2, 2371, 4128, 2),
                                          (4, 20003, 1184, 2), (3, 2050, 3076, 2), (1, 4100, 12288, 2), (4, 2048, 4096, 1), (2, 2051, 8192, 1), (1, 700, 2336, 1)])
def test_32_bit_products_of_up_to_four_rows(m, n, k, groups):
    """Whichever kernel: the bits that the same rows have beside others."""
    from llm_infer_rust_b200.kernels import ops
    from llm_infer_rust_b200.kernels.build import load_cuda_library
    assert load_cuda_library("gemm_f32.cu").b200_gemm_f32_pair_groups(m, n, k, 148) == groups
    for spread in (0.0, 4.0):
        a, w = _rnd(130, k) * torch.exp(spread * _rnd(130, k, seed=2)), _rnd(n, k, seed=1) * torch.exp(spread * _rnd(n, k, seed=3))
        got = ops.gemm_f32(a[:m].contiguous(), w)
        want, size = a[:m].double() @ w.double().t(), a[:m].double().abs() @ w.double().abs().t()
        assert ((got.double() - want).abs() <= (24 + 1 + k / 256 + 10) * 2.0 ** -24 * size).all()      # (as test_32_bit_products_in_three_terms)
        for rows in (8, 130):
            assert torch.equal(ops.gemm_f32(a[:rows].contiguous(), w)[:m], got)
    ops.check_errors(a.device)


# one kernel each: a few rows (three kinds), a cluster a tile, blocks that walk over tiles
@pytest.mark.parametrize("m,n,k", [(3, 1024, 4096), (3, 4100, 4096), (7, 1024, 4096), (300, 1024, 4096), (1024, 4096, 2048)])
def test_32_bit_products_whose_rows_are_all_nan_or_infinite(m, n, k):
    """Every element of such rows is summed again.  No block waits so long for it that another of its warps gives up, and the
    other rows keep their bits.  (A thread an element would take, by estimate, tens of milliseconds a tile.)"""
    from llm_infer_rust_b200.kernels import ops
    x, w = _rnd(m, k), _rnd(n, k, seed=1)
    plain = ops.gemm_f32(x, w)
    for bad in (float("nan"), float("inf")):
        a = x.clone()
        a[m // 3:] = bad
        got = ops.gemm_f32(a, w)
        torch.cuda.synchronize()
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        ops.gemm_f32(a, w, out=got)
        end.record()
        ops.check_errors(a.device)
        assert torch.equal(got[:m // 3], plain[:m // 3])
        assert got[m // 3:].isnan().all()                       # (infinities of both signs meet in every sum)
        # a NaN costs a pass over its row; an infinity one over its row and W's for every element, 1,000 cycles and 16 warps a block
        if bad != bad:
            assert begin.elapsed_time(end) < 20.0


def test_32_bit_products_of_a_head_each():
    from llm_infer_rust_b200.kernels import ops
    for rows in (3, 70):
        x, w = _rnd(rows, 4 * 24 + 5), _rnd(4, 19, 24, seed=2)      # column ranges of wider rows, not 16-byte aligned
        parts = x[:, 5:].reshape(rows, 4, 24).transpose(0, 1)
        got = ops.head_products(parts, w)
        want = torch.einsum("hrk,hnk->hrn", parts.double(), w.double())
        assert ((got.double() - want).abs() <= 2.0 ** -20 * (1 + want.abs().max())).all()


@pytest.mark.parametrize("dtype,width", [(torch.bfloat16, 1024), (torch.bfloat16, 1032), (torch.bfloat16, 4096), (torch.bfloat16, 16384),
                                         (torch.bfloat16, 16392), (torch.float32, 512), (torch.float32, 516), (torch.float32, 8192)])
def test_rms_norm_by_warps_by_blocks_and_beyond(dtype, width):
    from llm_infer_rust_b200.kernels import ops
    x, res, w = _rnd(5, width, dtype=dtype), _rnd(5, width, dtype=dtype, seed=1), _rnd(width, dtype=dtype, seed=2)
    s = x.double() + res.double()
    want = s / torch.sqrt((s * s).mean(-1, keepdim=True) + 1e-6) * w.double()
    kept = res.clone()
    got = ops.add_rms_norm(x, kept, w, 1e-6)
    bound = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20          # one rounding of the result; float sums of squares
    assert ((got.double() - want).abs() <= bound * want.abs() + 1e-6).all()
    assert torch.equal(kept, (x.float() + res.float()).to(dtype))
    rows = torch.tensor([4, 0, 4], dtype=torch.int32, device=DEV)
    alone = ops.rms_norm(x, w, 1e-6, rows=rows)
    xd = x.double()[[4, 0, 4]]
    want = xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert ((alone.double() - want).abs() <= bound * want.abs() + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,width,column", [(1, 8, 0), (3, 2048, 8), (2, 4104, 16), (5, 40, 3), (3, 12, 0)])
def test_gates_in_whole_and_in_broken_vectors(tokens, width, column, dtype):
    from llm_infer_rust_b200.kernels import ops
    packed, a = _rnd(tokens, column + width + 8, dtype=dtype, scale=4.0), _rnd(tokens, width, dtype=dtype, seed=1)
    want = a.double() * torch.sigmoid(packed[:, column:column + width].double())
    got = ops.sigmoid_gate_mul(a.clone(), packed, column)
    assert ((got.double() - want).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21) * want.abs() + 1e-9).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_gated_row_is_the_same_in_every_batch(dtype):
    """Few narrow rows take one element a thread, many take eight: to the bit the same."""
    from llm_infer_rust_b200.kernels import ops
    packed, a = _rnd(4200, 512, dtype=dtype, scale=4.0), _rnd(4200, 256, dtype=dtype, seed=1)
    many, few = ops.sigmoid_gate_mul(a.clone(), packed, 256), ops.sigmoid_gate_mul(a[:9].clone(), packed[:9], 256)
    assert torch.equal(many[:9], few)
    want = a.double() * torch.sigmoid(packed[:, 256:].double())
    assert ((many.double() - want).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21) * want.abs() + 1e-9).all()


@pytest.mark.parametrize("lengths", [[1 + (37 * i) % 200 for i in range(40)], [64] * 39 + [1], list(range(1, 75))])
def test_decoded_rows_of_many_lengths_in_several_waves(lengths):
    """More CTAs than SMs, rows listed in any order: every row is its own."""
    from llm_infer_rust_b200.kernels import ops
    H, G, D, page, n = 8, 4, 128, 16, len(lengths)
    pages = [-(-x // page) for x in lengths]
    first, width = [1 + sum(pages[:i]) for i in range(n)], max(pages)
    kc, vc = (_rnd(1 + sum(pages), G, page, D, dtype=torch.bfloat16, seed=s) for s in (3, 4))
    table = torch.zeros(n, width, dtype=torch.int32)
    for i in range(n):
        table[i, :pages[i]] = torch.arange(first[i], first[i] + pages[i])
    q = _rnd(n, H * D, dtype=torch.bfloat16, seed=5)
    out = torch.empty_like(q)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    ops.decode_attention(q, kc, vc, out, None, table.to(DEV), i32(list(range(n + 1))), i32(lengths), i32(list(range(n))), n, H, G, D, page,
                         None, D ** -0.5, 1)
    ops.check_errors(torch.device(DEV))
    for i in range(n):
        k, v = (c[first[i]:first[i] + pages[i]].transpose(1, 2).reshape(-1, G, D)[:lengths[i]].double().repeat_interleave(H // G, 1) for c in (kc, vc))
        s = torch.einsum("hd,jhd->hj", q[i].view(H, D).double(), k) * D ** -0.5
        want = torch.einsum("hj,jhd->hd", torch.softmax(s, 1), v)
        # a weight is rounded to 8 bits, and so is the result
        assert ((out[i].view(H, D).double() - want).abs() <= 2.0 ** -8 * (want.abs() + v.abs().amax(0))).all(), i


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv", [(16, 8), (5, 1)])
def test_a_token_between_projection_and_attention_is_the_same_in_every_batch(nh, nkv, dtype):
    """Few tokens take one head a lane group, more two, many four (the head count no multiple of it): to the bit the same."""
    from llm_infer_rust_b200.kernels import ops
    d, page, n = 128, 16, 3000
    x, pos = _rnd(n, (nh + 2 * nkv) * d, dtype=dtype), torch.arange(n, dtype=torch.int32, device=DEV)
    qw, kw = _rnd(d, dtype=dtype, seed=1), _rnd(d, dtype=dtype, seed=2)
    cos, sin = _rnd(n, d // 2, seed=3), _rnd(n, d // 2, seed=4)
    got = []
    for tokens in (n, 600, 300, 7):
        q = torch.empty(tokens, nh * d, dtype=dtype, device=DEV)
        kc, vc = (torch.zeros(n // page + 2, nkv, page, d, dtype=dtype, device=DEV) for _ in range(2))
        ops.qkv_post(x[:tokens], q, kc, vc, qw, kw, 1e-6, cos, sin, d, pos[:tokens], pos[:tokens] + page, nh, nkv, d)
        got.append((q[:7], kc[1, :, :7], vc[1, :, :7]))
    ops.check_errors(torch.device(DEV))
    assert all(torch.equal(a, b) for other in got[1:] for a, b in zip(got[0], other))
    rows = x[:7].double().view(7, nh + 2 * nkv, d)
    for h, (mine, w) in enumerate([(got[0][0].view(7, nh, d)[:, 0], qw), (got[0][1][0], kw)]):
        t = rows[:, h * nh]
        t = t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-6) * w.double()
        a, b, c, s = t[:, :64], t[:, 64:], cos[:7].double(), sin[:7].double()
        want = torch.cat([a * c - b * s, b * c + a * s], 1)
        # one rounding of the result; both products of a rotation carry a few of 2^-24
        assert ((mine.double() - want).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20) * (want.abs() + 1)).all()


def test_a_row_of_few_rows_experts_is_the_same_in_every_step():
    """Two rows take two columns a warp, 32 rows of two of eight experts one: to the bit the same (columns no multiple of a block's)."""
    from llm_infer_rust_b200.kernels import ops
    E, top, width, ff = 8, 2, 1032, 1544
    gu, dn = _rnd(E, 2 * ff, width, dtype=torch.bfloat16, scale=width ** -0.5), _rnd(E, width, ff, dtype=torch.bfloat16, seed=1, scale=ff ** -0.5)
    x, gains = _rnd(32, width, dtype=torch.bfloat16, seed=2), _rnd(32, top, seed=3).abs()
    choice = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(i))[:top] for i in range(32)]).to(torch.int32).to(DEV)
    many = ops.routed_experts(x, choice, gains, gu, dn)
    for n in (1, 2, 5):
        assert torch.equal(ops.routed_experts(x[:n], choice[:n], gains[:n], gu, dn), many[:n])
    for t in (0, 31):
        want = torch.zeros(width, dtype=torch.float64, device=DEV)
        for k in range(top):
            e = int(choice[t, k])
            g, u = (gu[e].double() @ x[t].double()).split(ff)
            want += gains[t, k].double() * (dn[e].double() @ (torch.nn.functional.silu(g) * u).bfloat16().double())
        # the hidden row is rounded to 8 bits, where a sum in 32 bits may fall on the other side
        assert ((many[t].double() - want).abs() <= 2.0 ** -8 * want.abs().max()).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("head_dim,ctas", [(16, 3), (32, 3), (48, 2), (64, 3), (128, 2)])
def test_all_sizes_prompt_attention_keeps_its_blocks_on_an_sm(head_dim, ctas, dtype):
    """A few registers more a thread and an SM holds a block less; long prompts then take up to twice the time."""
    from llm_infer_rust_b200.kernels import ops
    assert ops._attention(head_dim).b200_prefill_attention_ctas_per_sm(ops.F32 if dtype == torch.float32 else ops.BF16) >= ctas


@pytest.mark.parametrize("head_dim", [16, 32, 48, 64, 96, 128])
def test_32_bit_prompt_attention_keeps_its_numbers_in_registers(head_dim):
    """(One CTA an SM at every size; the float32 cases above are heads of 24, 40 and the like, which the all-sizes kernel keeps.)"""
    from llm_infer_rust_b200.kernels import ops
    assert ops._attention(head_dim).b200_prefill_split_local_bytes() == 0


# more steps than the grid has lane groups, with a rest; an odd count of heads (the last step has one); heads of 64 and 256 (8 and 32
# lanes); without norms, without tables, without a cache
@pytest.mark.parametrize("tokens,nh,nkv,d,norm,turn,store", [(1020, 16, 8, 128, True, True, True), (2500, 32, 8, 128, True, True, True),
                                                             (3001, 15, 5, 128, False, True, True), (6000, 9, 1, 64, True, True, False),
                                                             (1300, 8, 4, 256, True, False, True)])
def test_between_projection_and_attention_many_tokens_are_as_few(tokens, nh, nkv, d, norm, turn, store):
    from llm_infer_rust_b200.kernels import ops
    from llm_infer_rust_b200.kernels.build import load_entry_points
    steps = tokens * -(-(nh + 2 * nkv) // 2) * d // 8
    assert load_entry_points("qkv_post.cu").b200_qkv_post_walks(ops.BF16, steps)
    qkv = _rnd(tokens, (nh + 2 * nkv) * d, dtype=torch.bfloat16)
    w = [_rnd(d, dtype=torch.bfloat16, seed=s) for s in (1, 2)] if norm else [None, None]
    cos, sin = (_rnd(700, d // 2, seed=s) for s in (3, 4)) if turn else (None, None)
    gen = torch.Generator().manual_seed(5)
    pos = torch.randint(0, 700, (tokens,), generator=gen).int().to(DEV)
    slots = torch.randperm(tokens, generator=gen).int().to(DEV) + 16 if store else None
    if store:
        slots[::7] = 0                                          # padding rows
    out = []
    for cut in (tokens, 10):                                    # all at once, and ten tokens a call (the other kernel)
        k = torch.zeros(tokens // 16 + 3, nkv, 16, d, dtype=torch.bfloat16, device=DEV) if store else None
        v, q = torch.zeros_like(k) if store else None, torch.zeros(tokens, nh * d, dtype=torch.bfloat16, device=DEV)
        for at in range(0, tokens, cut):
            part = slice(at, at + cut)
            ops.qkv_post(qkv[part], q[part], k, v, w[0], w[1], 1e-6, cos, sin, d if turn else 0, pos[part],
                         slots[part] if store else None, nh, nkv, d)
        out.append([q] + ([k, v] if store else []))
    assert all(torch.equal(a, b) for a, b in zip(*out))
    ops.check_errors(qkv.device)


def test_many_tokens_refuse_slots_and_positions_outside():
    from llm_infer_rust_b200.kernels import ops
    tokens, nh, nkv, d = 1200, 16, 8, 128
    qkv, q = _rnd(tokens, (nh + 2 * nkv) * d, dtype=torch.bfloat16), torch.zeros(tokens, nh * d, dtype=torch.bfloat16, device=DEV)
    k = torch.zeros(80, nkv, 16, d, dtype=torch.bfloat16, device=DEV)
    v, cos, sin = torch.zeros_like(k), _rnd(1200, d // 2), _rnd(1200, d // 2)
    pos, slots = torch.arange(tokens, dtype=torch.int32, device=DEV), torch.arange(tokens, dtype=torch.int32, device=DEV) + 16
    for bad, where, what in ((1200, pos, "rotary"), (-1, pos, "rotary"), (80 * 16, slots, "slot"), (-5, slots, "slot")):
        kept = where[777].clone()
        where[777] = bad
        ops.qkv_post(qkv, q, k, v, None, None, 1e-6, cos, sin, d, pos, slots, nh, nkv, d)
        where[777] = kept
        with pytest.raises(ops.KernelError, match=what):
            ops.check_errors(qkv.device)


def _paged(lens, cached, nkv, d, page, seed=0):
    """Random pages of rows that hold ``cached`` + ``lens`` positions each: caches, block table, the rows' index arrays."""
    gen = torch.Generator().manual_seed(seed)
    total = [a + b for a, b in zip(lens, cached)]
    pages = [-(-t // page) for t in total]
    order, table, at = torch.randperm(sum(pages), generator=gen) + 1, torch.zeros(len(lens), max(pages), dtype=torch.int32), 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n
    k, v = (torch.randn(sum(pages) + 1, nkv, page, d, generator=gen).to(DEV) for _ in range(2))
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    return k, v, table.to(DEV), ints(starts), ints(total), ints(cached), ints(list(range(len(lens))))


def _attention_64(q, k, v, table, lens, cached, nh, nkv, d, page, scale, window=0, chunk=0, cap=0.0, sinks=None):
    out, at = [], 0
    for i, (n, p) in enumerate(zip(lens, cached)):
        t = n + p
        ks, vs = (c[table[i, :-(-t // page)].long()].double().permute(0, 2, 1, 3).reshape(-1, nkv, d)[:t].repeat_interleave(nh // nkv, 1)
                  for c in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[at:at + n].double().view(n, nh, d), ks) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        pos, key = torch.arange(p, t, device=DEV)[:, None], torch.arange(t, device=DEV)[None]
        hidden = (key > pos) | ((pos - key >= window) if window else False) | ((pos // chunk != key // chunk) if chunk else False)
        s = s.masked_fill(hidden, float("-inf"))
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None, None].expand(-1, n, 1)], 2)
        out.append(torch.einsum("hqk,khd->qhd", torch.softmax(s, -1)[:, :, :t], vs).reshape(n, -1))
        at += n
    return torch.cat(out)


# float32 portions on mma.sync: one key more than a quarter of a block (16), than a block (64) and than two; tiles with a rest; groups of
# 1, 2, 7, 16 and 40 (two chunks of heads); heads of 16, 48, 64, 96 and 128; page sizes of no power of two; windows and blocks inside
# a block of keys; caps and sinks; heads that only the other kernel takes (24: no multiple of 16)
@pytest.mark.parametrize("lens,cached,nh,nkv,d,page,form", [
    ([17], [0], 16, 8, 128, 16, {}), ([65, 1, 40], [0, 130, 3], 16, 8, 128, 16, {}), ([33], [96], 8, 8, 64, 16, {}),
    ([50], [10], 40, 1, 64, 4, {}), ([40], [0], 14, 2, 16, 16, {}), ([65], [3], 32, 2, 96, 3, {}), ([129], [0], 4, 4, 48, 16, {}),
    ([100], [30], 16, 8, 128, 16, dict(window=17)), ([100], [30], 16, 8, 128, 16, dict(chunk=40)),
    ([70], [30], 16, 8, 128, 16, dict(softcap=5.0)), ([64], [0], 16, 8, 64, 16, dict(sinks=True)), ([30], [20], 4, 2, 24, 16, {})])
def test_32_bit_prompt_attention(lens, cached, nh, nkv, d, page, form):
    from llm_infer_rust_b200.kernels import ops
    k, v, table, cu, total, prefix, rows = _paged(lens, cached, nkv, d, page)
    q, form = _rnd(sum(lens), nh * d, seed=3, scale=3.0), dict(form)
    window, scale = form.pop("window", None), d ** -0.5
    if form.pop("sinks", False):
        form["sinks"] = _rnd(nh, seed=4)

    def attend(q, lens, cu, total, prefix):
        out = torch.empty_like(q)
        ops.prefill_attention(q, k, v, out, table, cu, total, prefix, rows, len(lens), max(lens), nh, nkv, d, page, window, scale, **form)
        return out
    got = attend(q, lens, cu, total, prefix)
    want = _attention_64(q, k, v, table, lens, cached, nh, nkv, d, page, scale, window or 0, form.get("chunk", 0), form.get("softcap", 0.0),
                         form.get("sinks"))
    # scores of up to 3 x 5 with sums of d terms in 32 bits: 2^-24 x 15 x (2 + log2 d) in the exponent, as much again in the sums
    assert (got.double() - want).abs().max() <= 2.0 ** -24 * 400 * v.abs().max()
    if len(lens) == 1:                                          # the same bits however the portion is cut
        parts, ints = [], lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
        cuts = [0, 1, lens[0] // 2, lens[0]]
        for lo, hi in zip(cuts, cuts[1:]):
            parts.append(attend(q[lo:hi].contiguous(), [hi - lo], ints(0, hi - lo), ints(cached[0] + hi), ints(cached[0] + lo)))
        if d != 24 or not window and not form.get("chunk"):     # (d = 24: the other kernel, whose first block follows the first query's window)
            assert torch.equal(torch.cat(parts), got)


@pytest.mark.parametrize("exponent", [-105, -118])
def test_32_bit_prompt_attention_of_very_small_values(exponent):
    """Above and below 2^-110, where a third term no longer has all its bits."""
    from llm_infer_rust_b200.kernels import ops
    lens, cached, nh, nkv, d, page = [50], [30], 4, 2, 64, 16
    k, v, table, cu, total, prefix, rows = _paged(lens, cached, nkv, d, page)
    q, v = _rnd(50, nh * d, seed=3), (v.abs() + 1.0) * 2.0 ** exponent
    out = torch.empty_like(q)
    ops.prefill_attention(q, k, v, out, table, cu, total, prefix, rows, 1, 50, nh, nkv, d, page, None, d ** -0.5)
    want = _attention_64(q, k, v, table, lens, cached, nh, nkv, d, page, d ** -0.5)
    # values of one sign: as test_32_bit_prompt_attention relative to the result, and the products' roundings below 2^-126
    assert ((out.double() - want).abs() <= 2.0 ** -24 * 400 * want + 200 * 2.0 ** -150).all()


def test_32_bit_prompt_attention_of_infinities():
    """Infinities and NaN of queries, keys and values come out where a plain softmax puts them."""
    from llm_infer_rust_b200.kernels import ops
    lens, cached, nh, nkv, d, page = [90], [0], 4, 2, 64, 16
    k, v, table, cu, total, prefix, rows = _paged(lens, cached, nkv, d, page)
    q = _rnd(90, nh * d, seed=3)
    at = lambda position: (table[0, position // page].item(), position % page)
    for what in ("value", "key", "query"):
        kk, vv, qq = k.clone(), v.clone(), q.clone()
        if what == "value":
            vv[at(37)[0], 1, at(37)[1], 7] = float("inf")
        elif what == "key":
            kk[at(50)[0], 0, at(50)[1], 3] = float("nan")
        else:
            qq[66, 5] = float("-inf")
        out = torch.empty_like(qq)
        ops.prefill_attention(qq, kk, vv, out, table, cu, total, prefix, rows, 1, 90, nh, nkv, d, page, None, d ** -0.5)
        want = _attention_64(qq, kk, vv, table, lens, cached, nh, nkv, d, page, d ** -0.5)
        if what == "value":       # (a key that is not visible has the weight zero, and zero times infinity is a NaN in both kernels' blocks of keys)
            seen = slice(37, 90)
            assert torch.equal(out[seen].isinf(), want[seen].isinf()) and out[seen].isinf().sum() == 53 * 2
            assert out[:32].isfinite().all()
        else:
            assert torch.equal(out.isnan(), want.isnan()) and out.isnan().any() and not out.isnan().all()


@pytest.mark.parametrize("what", ["key", "query", "small"])
def test_32_bit_prompt_attention_beside_rows_that_are_done_again(what):
    """Rows without a finite result, or with a very small one, leave the bits of the rows and heads in their tile as they are."""
    from llm_infer_rust_b200.kernels import ops
    nh, nkv, d, page = 4, 2, 64, 16
    k, v, table, _, _, _, rows = _paged([90], [0], nkv, d, page)
    q = _rnd(90, nh * d, seed=3)
    ints = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)

    def attend(q, first=0):
        out = torch.empty_like(q)
        ops.prefill_attention(q, k, v, out, table, ints(0, len(q)), ints(first + len(q)), ints(first), rows, 1, len(q), nh, nkv, d, page, None, d ** -0.5)
        return out
    if what == "small":                                         # the first row sees nothing but the first key
        v[table[0, 0].item(), :, 0] *= 2.0 ** -118
        got = attend(q)
        assert 0.0 < got[0].abs().max() < 2.0 ** -80 and got[1:].abs().amin(1).min() > 2.0 ** -80
        assert torch.equal(got[1:], attend(q[1:].contiguous(), 1))
        return
    plain = attend(q)
    if what == "key":
        k[table[0, 50 // page].item(), 0, 50 % page, 3] = float("nan")
    else:
        q[66, 5] = float("-inf")
    got = attend(q).view(90, nh, d)
    other = ~got.isnan()
    assert other.view(90, -1).sum().item() == ((50 * nh + 40 * 2) if what == "key" else (90 * nh - 1)) * d
    assert torch.equal(got[other], plain.view(90, nh, d)[other])
