"""The further forms of the tcgen05 prompt attention (keys and values of 128: soft-cap, weights in two terms, blocks of
positions, sinks, windows, the difference of two maps) against the plain softmax in 64 bits, at the edges of its tiles of 128
query vectors and blocks of 128 keys."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D = 128


def _plain(q, k, v, scale, cap, window, chunk, sinks, first):
    """q [n, H, D] at positions first .., k and v [T, G, D]: float64 [n, H, D]."""
    n, H = q.shape[:2]
    rep = H // k.shape[1]
    s = torch.einsum("ihd,jhd->hij", q.double(), k.double().repeat_interleave(rep, 1)) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    i, j = torch.arange(first, first + n)[:, None], torch.arange(k.shape[0])[None]
    seen = j <= i
    if window:
        seen &= i - j < window
    if chunk:
        seen &= i // chunk == j // chunk
    s = s.masked_fill(~seen, float("-inf"))
    if sinks is not None:
        s = torch.cat([s, sinks.double()[:, None, None].expand(H, n, 1)], 2)
    return torch.einsum("hij,jhd->ihd", torch.softmax(s, 2)[:, :, :k.shape[0]], v.double().repeat_interleave(rep, 1))


FORMS = [dict(cap=5.0), dict(), dict(cap=3.0, window=100), dict(window=17), dict(chunk=130), dict(chunk=48, sinks=True), dict(sinks=True),
         dict(difference=(0.6, 0.65, 1e-5)), dict(difference=(0.6, 0.65, 1e-5), window=129)]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(f) or "split")
@pytest.mark.parametrize("H,G,portions", [(4, 2, [128, 1, 130, 65]), (2, 2, [256, 257, 1]), (8, 1, [300]), (16, 1, [16, 17, 240]), (4, 1, [64, 3, 400])])
def test_forms_against_the_plain_softmax(H, G, portions, form):
    from llm_infer_rust_b200.kernels import ops
    cap, window, chunk = form.get("cap", 0.0), form.get("window"), form.get("chunk")
    difference = form.get("difference")
    if difference and (H // G) % 2:
        pytest.skip("a difference needs pairs of maps")
    page, T, dev = 16, sum(portions), "cuda"
    g = torch.Generator().manual_seed(T + H)
    q, k, v = (torch.randn(T, n, D, generator=g).bfloat16() for n in (H, G, G))
    for i in (T - 1, T // 2, 130 % T):                 # a key just outside the mask, one at its edge and the first fit best
        lo = max(0, i - window + 1) if window else i - i % chunk if chunk else 0
        for j, boost in ((max(0, lo - 1), 3.0), (lo, 2.0), (0, 2.5)):
            k[j, 0] = (boost * q[i, 0].float() / q[i, 0].float().norm() * 4.0).bfloat16()
    sinks = torch.linspace(-2.0, 4.0, H) if form.get("sinks") else None
    pages = -(-T // page)
    order = torch.randperm(pages, generator=g) + 1
    caches = [torch.full((pages + 1, G, page, D), 77.0, dtype=torch.bfloat16) for _ in range(2)]     # stale values beyond
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    scale, at, heads = 0.3, 0, H // 2 if difference else H
    for n in portions:
        for cache, rows in zip(caches, (k, v)):
            for p in range(at, at + n):
                cache[order[p // page], :, p % page] = rows[p]
        kc, vc = (c.to(dev) for c in caches)
        out = torch.full((n, heads * D), float("nan"), dtype=torch.bfloat16, device=dev)
        before = ops.tcgen05_shaped_launches()
        ops.prefill_attention(q[at:at + n].reshape(n, -1).to(dev).contiguous(), kc, vc, out, order.to(torch.int32).reshape(1, -1).to(dev),
                              i32([0, n]), i32([at + n]), i32([at]), i32([0]), 1, n, H, G, D, page, window, scale, v_head_dim=D,
                              softcap=cap, precise_weights=True, chunk=chunk, sinks=None if sinks is None else sinks.to(dev),
                              difference=difference)
        ops.check_errors(torch.device(dev))
        assert ops.tcgen05_shaped_launches() - before == (1 if n * (H // G) >= 256 else 0)
        want = _plain(q[at:at + n], k[:at + n], v[:at + n], scale, cap, window, chunk, sinks, at)
        slack = 2.0 ** -13 * v.float().abs().max().item()           # weights of 16 bits, sums and exponents in 32
        if difference:
            lam, gain, eps = difference
            o = want[:, 0::2] - lam * want[:, 1::2]
            f = gain / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)
            want, slack = o * f, 4 * slack * f                      # two maps, and the root that their error moves
        got = out.cpu().double().reshape(n, heads, D)
        assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + slack).all()      # the stored value is rounded to 8 bits
        at += n


@pytest.mark.parametrize("scale", [0.0, -0.2, 0.3])
@pytest.mark.parametrize("H,G,rows", [(4, 4, 40), (16, 8, 1)])
def test_a_scale_of_any_sign(H, G, rows, scale):
    """Plain prompts at sizes where scale > 0 takes two tiles a CTA (40 rows) and one: with scale 0 every visible key weighs the
    same, with scale < 0 the worst fitting one weighs most."""
    from llm_infer_rust_b200.kernels import ops
    page, n, dev = 16, 300, "cuda"
    g = torch.Generator().manual_seed(rows)
    q = torch.randn(rows * n, H, D, generator=g).bfloat16()
    k, v = (torch.randn(rows, n, G, D, generator=g).bfloat16() for _ in range(2))
    pages = -(-n // page)
    caches = []
    for x in (k, v):
        c = torch.zeros(1 + rows * pages, G, page, D, dtype=torch.bfloat16)
        c[1:] = torch.nn.functional.pad(x, (0, 0, 0, 0, 0, pages * page - n)).reshape(rows * pages, page, G, D).transpose(1, 2)
        caches.append(c.to(dev))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    out = torch.empty(rows * n, H * D, dtype=torch.bfloat16, device=dev)
    before = ops.tcgen05_attention_launches()
    ops.prefill_attention(q.reshape(rows * n, -1).to(dev), *caches, out, i32([[1 + r * pages + p for p in range(pages)] for r in range(rows)]),
                          i32([r * n for r in range(rows + 1)]), i32([n] * rows), i32([0] * rows), i32(list(range(rows))), rows, n, H, G, D, page,
                          None, scale)
    ops.check_errors(torch.device(dev))
    took = tuple(b - a for a, b in zip(before, ops.tcgen05_attention_launches()))
    assert took == ((0, 0) if scale <= 0 else (0, 1) if rows > 1 else (1, 0))
    for r in (0, rows - 1):
        want = _plain(q[r * n:(r + 1) * n], k[r], v[r], scale, 0.0, None, None, None, 0)
        got = out[r * n:(r + 1) * n].cpu().double().reshape(n, H, D)
        # a weight is rounded to 8 bits, and so is the result
        assert ((got - want).abs() <= 2.0 ** -8 * (want.abs() + v[r].float().abs().max().item())).all()


@pytest.mark.parametrize("form", [dict(), dict(precise_weights=True, softcap=5.0), dict(precise_weights=True, difference=(0.6, 0.65, 1e-5))],
                         ids=lambda f: "-".join(f) or "plain")
def test_an_output_between_16_byte_boundaries(form):
    """The output may be a view that begins 4 or 8 bytes into its storage: another kernel serves it, to the same result."""
    from llm_infer_rust_b200.kernels import ops
    H, G, page, n, dev = 4, 2, 16, 300, "cuda"
    g = torch.Generator().manual_seed(3)
    q = torch.randn(n, H * D, generator=g).bfloat16().to(dev)
    kc, vc = (torch.randn(20, G, page, D, generator=g).bfloat16().to(dev) for _ in range(2))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    width = H * D // 2 if "difference" in form else H * D
    outs = []
    for skip in (0, 2, 4):                                # elements of two bytes
        out = torch.full((n * width + 8,), float("nan"), dtype=torch.bfloat16, device=dev)[skip:skip + n * width].view(n, width)
        before = sum(ops.tcgen05_attention_launches()) + ops.tcgen05_shaped_launches()
        ops.prefill_attention(q, kc, vc, out, i32([list(range(1, 20))]), i32([0, n]), i32([n]), i32([0]), i32([0]), 1, n, H, G, D, page, None,
                              0.2, v_head_dim=D, **form)
        ops.check_errors(torch.device(dev))
        assert sum(ops.tcgen05_attention_launches()) + ops.tcgen05_shaped_launches() - before == (0 if skip else 1)
        outs.append(out.double())
    assert torch.equal(outs[1], outs[2])
    # two roundings to 8 bits apart, and (plain) weights of 8 bits on both sides; a difference's root moves with its maps' error
    assert (outs[0] - outs[1]).abs().max() <= (2.0 ** -7 + (2.0 ** -8 if not form else 2.0 ** -10)) * vc.double().abs().max()


SEVERAL = [dict(cap=5.0), dict(chunk=130, sinks=True), dict(window=129, difference=(0.6, 0.65, 1e-5)), dict(cap=5.0, sinks=True),
           dict(window=100, sinks=True), dict(chunk=48)]


@pytest.mark.parametrize("precise", [True, False], ids=["two-terms", "one-term"])
@pytest.mark.parametrize("form", SEVERAL, ids="-".join)
@pytest.mark.parametrize("H,G", [(4, 2), (4, 1)])
def test_forms_over_rows_of_all_lengths(H, G, form, precise):
    """Several rows in one launch, named in another order than the batch's, with cached tokens before them, among them rows with
    nothing in most of the grid's tiles; weights in two bfloat16 terms and in one."""
    from llm_infer_rust_b200.kernels import ops
    cap, window, chunk, difference = form.get("cap", 0.0), form.get("window"), form.get("chunk"), form.get("difference")
    rows, page, dev = [(0, 700), (300, 333), (5, 1), (0, 128)], 16, "cuda"
    g = torch.Generator().manual_seed(H)
    n = sum(r[1] for r in rows)
    q = torch.randn(n, H, D, generator=g).bfloat16()
    k, v = ([torch.randn(a + b, G, D, generator=g).bfloat16() for a, b in rows] for _ in range(2))
    pages = [-(-(a + b) // page) for a, b in rows]
    order = (torch.randperm(sum(pages), generator=g) + 1).tolist()
    caches = [torch.full((sum(pages) + 1, G, page, D), 77.0, dtype=torch.bfloat16) for _ in range(2)]      # stale values beyond
    table = torch.zeros(len(rows), max(pages), dtype=torch.int32)
    for r, (a, b) in enumerate(rows):
        mine = [order.pop() for _ in range(pages[r])]
        table[r, :pages[r]] = torch.tensor(mine, dtype=torch.int32)
        for cache, x in zip(caches, (k[r], v[r])):
            for p in range(a + b):
                cache[mine[p // page], :, p % page] = x[p]
    sinks = torch.linspace(-2.0, 4.0, H) if form.get("sinks") else None
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    first, heads = [0, 700, 1033, 1034, 1162], H // 2 if difference else H
    out = torch.full((n, heads * D), float("nan"), dtype=torch.bfloat16, device=dev)
    before = ops.tcgen05_shaped_launches()
    ops.prefill_attention(q.reshape(n, -1).to(dev), *(c.to(dev) for c in caches), out, table.to(dev), i32(first), i32([a + b for a, b in rows]),
                          i32([a for a, _ in rows]), i32([2, 0, 3, 1]), 4, 700, H, G, D, page, window, 0.3, v_head_dim=D, softcap=cap,
                          precise_weights=precise, chunk=chunk, sinks=None if sinks is None else sinks.to(dev), difference=difference)
    ops.check_errors(torch.device(dev))
    assert ops.tcgen05_shaped_launches() - before == 1
    for r, (a, b) in enumerate(rows):
        at = slice(first[r], first[r + 1])
        want = _plain(q[at], k[r], v[r], 0.3, cap, window, chunk, sinks, a)
        # weights of 16 bits or of 8, sums and exponents in 32
        slack = 2.0 ** (-13 if precise else -8) * v[r].float().abs().max().item()
        if difference:
            lam, gain, eps = difference
            o = want[:, 0::2] - lam * want[:, 1::2]
            f = gain / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)
            want, slack = o * f, 4 * slack * f                      # two maps, and the root that their error moves
        got = out[at].cpu().double().reshape(b, heads, D)
        assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + slack).all(), r
