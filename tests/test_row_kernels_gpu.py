"""Edges of the kernels that walk a step's rows: sizes at which a thread holds its whole share in registers and just beyond, sizes without
16-byte accesses, and the numbers of tokens at which another form of a kernel takes over (equal bits: a token does not show its step)."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H", [4, 127, 2048, 2052, 8192, 8196, 10240, 2050])
def test_layer_norm_at_the_edges_of_a_thread(H):
    """Against 64 bits. The bound is 2e-6 of the largest value: sixteen roundings of a 32-bit result (three partial sums, two means, the scale)."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(H)
    h, parts = torch.randn(5, H, generator=g) * 2 + 0.5, torch.randn(3, 5, H, generator=g)
    w, b = torch.randn(H, generator=g), torch.randn(H, generator=g)
    out, hd = torch.empty(5, H, device=DEV), h.to(DEV)
    ops.layernorm(hd, w.to(DEV), b.to(DEV), 1e-5, out, partials=parts.to(DEV))
    x = h.double() + parts.double().sum(0)
    d = x - x.mean(-1, keepdim=True)
    want = d / torch.sqrt((d * d).mean(-1, keepdim=True) + 1e-5) * w.double() + b.double()
    assert (out.cpu().double() - want).abs().max() <= 2e-6 * float(want.abs().max())
    assert (hd.cpu().double() - x).abs().max() <= 1e-6 * float(x.abs().max())
    alone = torch.empty(1, H, device=DEV)
    ops.layernorm(h[3:4].to(DEV), w.to(DEV), b.to(DEV), 1e-5, alone, partials=parts[:, 3:4].contiguous().to(DEV))
    assert torch.equal(alone[0], out[3])


@pytest.mark.parametrize("F", [5, 1020, 8192, 8196, 9001, 12288])
def test_polynorm_at_the_edges_of_a_thread(F):
    """Against 64 bits, within 4e-6 of the largest value (six partial sums, cubed: their roundings three times over, a mean, the result's own)."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(F)
    up = torch.randn(6, 4, F, generator=g) * 0.4                     # (more partial buffers than are requested together)
    a, b, c, e = 0.7, -0.3, 0.2, 0.05
    out = torch.empty(4, F, device=DEV)
    ops.polynorm(up.to(DEV), out, (a, b, c, e), 1e-5)
    z = up.double().sum(0)
    n = lambda y: y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5)
    want = a * n(z) + b * n(z ** 2) + c * n(z ** 3) + e
    assert (out.cpu().double() - want).abs().max() <= 4e-6 * float(want.abs().max())


@pytest.mark.parametrize("bw,B", [(128, 2), (100, 3), (10, 2), (33, 1), (260, 1), (16, 3), (272, 1)])
def test_gates_do_not_show_the_number_of_tokens(bw, B):
    """Both kernels of the gates, and one and four rows a block of the convolution: the bits of 1 to 257 tokens in those of 300."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(bw)
    C, n, K = bw * B, 300, 4
    dev = lambda *s, k=0.3: (torch.randn(*s, generator=g) * k).to(DEV)
    proj = dev(2, n, 2 * C)
    xb, yb, rb, ib, lam, taps, cb = dev(C), dev(C), dev(C), dev(C), dev(C) - 3.0, dev(C, K), dev(C)
    gate_w = dev(B, bw, 2 * bw).bfloat16()
    pos, slot = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    state = torch.zeros(1, K, C, device=DEV)

    def run(m):
        p = proj[:, :m].contiguous()
        u, a, d, y = (torch.empty(m, C, device=DEV) for _ in range(4))
        ops.rglru_conv(p, xb, taps, cb, pos[:m], slot[:m], state, u)
        ops.rglru_gates(gate_w, rb, ib, lam, yb, u, p, a, d, y)
        return u, a, d, y

    whole = run(n)
    for m in (1, 8, 128, 129, 257):
        for x, w in zip(run(m), whole):
            assert torch.equal(x, w[:m]), m


@pytest.mark.parametrize("D,rot", [(64, 32), (64, 8), (24, 8), (64, 64), (20, 4), (64, 0)])
def test_rotation_of_a_part_of_the_head(D, rot):
    """The 16-byte form (head and rotated part multiples of eight) and the single-element one against the rotation itself, in 32 bits."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(D + rot)
    n, Hq, Hkv, page = 7, 5, 2, 16
    qk = torch.randn(2, n, (Hq + Hkv) * D, generator=g)
    pos = torch.arange(3, 3 + n, dtype=torch.int32)
    angle = pos.float()[:, None] * torch.rand(max(rot // 2, 1), generator=g)[None]
    table = torch.zeros(16, max(rot // 2, 1), 2)
    table[3:3 + n] = torch.stack([angle.cos(), angle.sin()], -1)
    q_out = torch.empty(n, Hq * D, device=DEV)
    cache = torch.zeros(2, 2, Hkv, page, D, device=DEV)
    ops.rope_append(qk.to(DEV), pos.to(DEV), torch.zeros(n, dtype=torch.int32, device=DEV), table.to(DEV), rot, q_out, cache,
                    torch.tensor([[1]], dtype=torch.int32, device=DEV), Hq, Hkv, D, values_from_keys=True)
    x = qk.sum(0).view(n, Hq + Hkv, D)
    c, s = angle.cos()[:, None, :rot // 2], angle.sin()[:, None, :rot // 2]
    u, v = x[..., :rot // 2], x[..., rot // 2:rot]
    turned = torch.cat([u * c - v * s, v * c + u * s, x[..., rot:]], -1)
    assert (q_out.cpu() - turned[:, :Hq].reshape(n, -1)).abs().max() <= 1e-5
    assert (cache[1, 0, :, 3:3 + n].cpu().transpose(0, 1) - turned[:, Hq:]).abs().max() <= 1e-5
    assert torch.equal(cache[1, 1, :, 3:3 + n].cpu().transpose(0, 1), x[:, Hq:])


@pytest.mark.parametrize("M,K", [(1, 8), (149, 264), (2369, 248), (5000, 2056), (4737, 8192), (40, 12288)])
@pytest.mark.parametrize("wdtype", [torch.bfloat16, torch.float32])
def test_a_few_tokens_as_a_stream_over_the_weights(M, K, wdtype):
    """One to four tokens, features around the number of warps, rows that end within a piece: the bits of the tiles that many tokens take, and
    64 bits within K roundings of the sum of the products' magnitudes."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(M + K)
    w, x = (torch.randn(M, K, generator=g) * 0.1).to(wdtype).to(DEV), torch.randn(40, K, generator=g).to(DEV)
    tiles = torch.empty(40, M, device=DEV)
    ops.gemm_f32(x, w, tiles)
    for n in (1, 2, 3, 4):
        out = torch.full((n, M), 0.5, device=DEV)
        ops.gemm_f32(x[:n].contiguous(), w, out)
        assert torch.equal(out, tiles[:n])
        ops.gemm_f32(x[:n].contiguous(), w, out, accumulate=True)
        assert torch.equal(out, tiles[:n] + tiles[:n])
    xd, wd = x[:4].double(), w.double()
    assert ((tiles[:4].double() - xd @ wd.T).abs() <= (K / 32 + 40) * 2.0 ** -24 * (xd.abs() @ wd.abs().T)).all()


@pytest.mark.parametrize("window,keep,sinks", [(0, 0, False), (100, 0, True), (64, 5, True), (1, 0, False)])
def test_masked_attention_of_two_row_groups_a_block(window, keep, sinks):
    """Latent rows of 512 and 16 heads: a step of 410 tokens (two tokens a block; entries of odd lengths, one of which continues) in the bits
    of the same tokens in steps of at most 99 (a token a block), and the rows against the sum in 64 bits."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(window + keep)
    H, D, page, scale = 16, 512, 32, 0.05
    old, new = [0, 70], [333, 77]                                    # cached tokens in front, tokens of the step
    pages = (torch.randn(2 * 16, 1, 1, page, D, generator=g) * 0.5).bfloat16().to(DEV)
    table = torch.randperm(32, generator=g).view(2, 16).int().to(DEV)
    q = torch.randn(sum(new), H * D, generator=g).bfloat16().to(DEV)
    sink = torch.randn(H, generator=g).to(DEV) if sinks else None

    def run(rows, entries):
        meta = torch.tensor([[e[k] for e in entries] for k in range(4)], dtype=torch.int32, device=DEV)
        out = torch.empty(rows.shape[0], H * D, dtype=torch.bfloat16, device=DEV)
        ops.masked_attention_tiles(rows, out, pages, table, meta, len(entries), None, sink, H, 1, D, D, window, keep, scale)
        return out

    whole = run(q, [(0, 0, new[0], old[0]), (1, new[0], new[1], old[1])])
    first = 0
    for slot in (0, 1):
        keys = pages[table[slot].long(), 0, 0].reshape(-1, D).double()
        for a in range(0, new[slot], 99):
            n = min(99, new[slot] - a)
            part = run(q[first + a:first + a + n].contiguous(), [(slot, 0, n, old[slot] + a)])
            assert torch.equal(part, whole[first + a:first + a + n])
        i, j = torch.arange(new[slot], device=DEV)[:, None] + old[slot], torch.arange(keys.shape[0], device=DEV)[None]
        seen = (j <= i) & ((i - j < window) | (j < keep)) if window else j <= i
        s = torch.einsum("ihd,jd->hij", q[first:first + new[slot]].double().view(-1, H, D), keys) * scale
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.double().view(H, 1, 1).expand(H, new[slot], 1)], -1)
        want = torch.einsum("hij,jd->ihd", torch.softmax(s, -1)[..., :keys.shape[0]], keys).reshape(new[slot], -1)
        # half a step of bfloat16 of the largest value, and what the 32-bit exponentials leave
        assert (whole[first:first + new[slot]].double() - want).abs().max() <= 2.0 ** -8 * float(want.abs().max())
        first += new[slot]


@pytest.mark.parametrize("H", [2048, 2052, 4096, 8192, 8200, 1024, 516])
def test_rms_norm_does_not_show_its_form(H):
    """Four blocks a row (up to 64 rows behind several partial buffers), a block a row with twelve and with six buffers requested together, and
    half the threads for a row behind one buffer (here as two, the second zero, in the other forms): the same bits."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(H)
    n, w = 200, (1 + 0.1 * torch.randn(H, generator=g)).bfloat16().to(DEV)
    h, parts = torch.randn(n, H, generator=g).to(DEV), torch.randn(9, n, H, generator=g).to(DEV)
    zero = torch.zeros(1, n, H, device=DEV)
    for partials, alone in ((parts, None), (torch.cat([parts[:1], zero]), parts[:1])):
        def run(m, p, dtype):
            hd, out = h[:m].clone(), torch.empty(m, H, dtype=dtype, device=DEV)
            ops.rmsnorm(hd, w, 1e-5, out, partials=p[:, :m].contiguous())
            return hd, out
        for dtype in (torch.bfloat16, torch.float32):
            whole = run(n, partials, dtype)
            for m in (1, 64, 65, 148):
                for x, y in zip(run(m, partials, dtype), whole):
                    assert torch.equal(x, y[:m]), m
            if alone is not None:
                for x, y in zip(run(n, alone, dtype), whole):
                    assert torch.equal(x, y)
    x = h.double() + parts.double().sum(0)
    want = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double()
    out = torch.empty(64, H, device=DEV)
    ops.rmsnorm(h[:64].clone(), w, 1e-5, out, partials=parts[:, :64].contiguous())
    assert (out.double() - want[:64]).abs().max() <= 2e-6 * float(want.abs().max())      # sixteen roundings of a 32-bit result


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("window,keep", [(0, 0), (64, 5)])
def test_rows_never_meet_keys_they_do_not_see(bad, window, keep):
    """Two tokens a block share staged keys: the one in front does not see the other's latent, the other has one key less at the window's
    start. Latents that are no numbers change no row that does not see them, alone in a block or as one of two."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(window)
    H, D, page, n = 16, 512, 32, 400
    pages = (torch.randn(13, 1, 1, page, D, generator=g) * 0.5).bfloat16().to(DEV)
    table = torch.arange(13, dtype=torch.int32, device=DEV)[None]
    q = torch.randn(n, H * D, generator=g).bfloat16().to(DEV)

    def run(cache, first, count):
        meta = torch.tensor([[0], [0], [count], [first]], dtype=torch.int32, device=DEV)
        out = torch.empty(count, H * D, dtype=torch.bfloat16, device=DEV)
        ops.masked_attention_tiles(q[first:first + count].contiguous(), out, cache, table, meta, 1, None, None, H, 1, D, D, window, keep, 0.05)
        return out

    i = torch.arange(n, device=DEV)
    for key in (101, 154, 399):                     # the second and the first token of a block, the last of all
        damaged = pages.clone()
        damaged[key // page, 0, 0, key % page] = bad
        sees = (i >= key) & ((i - key < window) | (key < keep)) if window else i >= key
        for first, count in ((0, n), (90, 99), (301, 99)):
            clean, got, seen = run(pages, first, count), run(damaged, first, count), sees[first:first + count]
            assert torch.equal(got[~seen], clean[~seen]) and torch.isfinite(clean).all()
            assert not torch.isfinite(got[seen].float()).all() or not seen.any()


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("lengths", [[2, 0], [1, 3, 0, 0], [1, 1, 1]])
def test_recurrence_with_as_many_tokens_as_entries(gated, lengths):
    """The kernel of single tokens is chosen by the number of tokens and entries alone: entries without a token and entries of several give
    the bits of each entry's tokens in a step of their own."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(len(lengths))
    H, D, V, E, n = 2, 40, 36, len(lengths), len(lengths)
    rows, width = [sum(lengths[:i]) for i in range(E)], 3 * H * D + H * V
    act = torch.rand(n, width, generator=g).to(DEV)
    before = torch.randn(E, H, D, V, generator=g).to(DEV)

    def run(x, entries, state):
        meta = torch.tensor([[e[k] for e in entries] for k in range(4)], dtype=torch.int32, device=DEV)
        out = torch.zeros(x.shape[0], H * V, device=DEV)
        if gated:
            ops.gated_scan(x, 0, H * D, 2 * H * D, 3 * H * D, meta, len(entries), state, out, H, D, V)
        else:
            ops.lightning_scan(x, 0, H * D, 3 * H * D, meta, len(entries), torch.tensor([0.9, 0.99], device=DEV), state, out, H, D, V, torch.empty_like(x))
        return out

    state, alone = before.clone(), before.clone()
    out = run(act, [(i, rows[i], lengths[i], 5) for i in range(E)], state)
    for i in range(E):
        for t in range(lengths[i]):
            r = rows[i] + t
            assert torch.equal(run(act[r:r + 1].contiguous(), [(i, 0, 1, 5 + t)], alone)[0], out[r])
    assert torch.equal(state, alone)


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("H,D,tokens", [(1, 64, 511), (1, 64, 512), (4, 96, 255), (4, 96, 256), (8, 40, 127), (8, 40, 128), (8, 128, 31), (8, 128, 32), (12, 100, 15),
                                        (12, 100, 16), (12, 64, 15), (12, 64, 16), (12, 32, 63), (12, 32, 64), (18, 200, 20), (19, 200, 20)])
def test_recurrence_that_starts_early_or_behind_the_kernel_in_front(H, D, tokens, gated):
    """Launches on both sides of the lines between the two starts, their rows written by the kernel in front over NaN: the bits of portions of
    at most ten tokens."""
    from stride_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(H * D + tokens)
    V, HD, HV = 64, H * D, H * 64
    proj = torch.randn((1, tokens, 2 * HD + HV), device=DEV, generator=g) * 0.3
    lower, zero = torch.rand(HD, device=DEV, generator=g) * 0.5, torch.zeros(HD, device=DEV)
    decay = torch.rand(H, device=DEV, generator=g) * 0.5 + 0.4

    def run(first, count, state):
        act = torch.full((count, (3 if gated else 2) * HD + HV), float("nan"), device=DEV)
        meta = torch.tensor([[0], [0], [count], [first]], dtype=torch.int32, device=DEV)
        out = torch.zeros((count, HV), device=DEV)
        part = proj[:, first:first + count].contiguous()
        torch.cuda.synchronize()
        if gated:
            ops.hgrn2_activate(part, zero, lower, act, HD, HV)
            ops.gated_scan(act, 0, HD, 2 * HD, 3 * HD, meta, 1, state, out, H, D, V)
        else:
            ops.lightning_scan(part, 0, HD, 2 * HD, meta, 1, decay, state, out, H, D, V, act)
        return out

    whole, cut = (torch.full((1, H, D, V), float("nan"), device=DEV) for _ in range(2))
    out = run(0, tokens, whole)
    assert torch.isfinite(out).all()
    assert torch.equal(out, torch.cat([run(a, min(10, tokens - a), cut) for a in range(0, tokens, 10)])) and torch.equal(whole, cut)


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("D,tokens", [(144, 40), (144, 1), (40, 40), (40, 1), (16, 20)])
def test_recurrence_with_an_infinite_value(D, tokens, gated):
    """Key sizes that do not fill the lanes: an infinite value makes its own column infinite from its token on (all keys, queries and states
    are positive here) and nothing else; the elements that pad the keys add zeros."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(D)
    H, V = 2, 36
    act = 0.1 + torch.rand(tokens, 3 * H * D + H * V, generator=g)
    at, column = tokens // 2, 7
    act[at, 3 * H * D + column] = float("inf")
    meta = torch.tensor([[0], [0], [tokens], [3]], dtype=torch.int32, device=DEV)
    state, out = torch.rand(1, H, D, V, generator=g).to(DEV), torch.zeros(tokens, H * V, device=DEV)
    if gated:
        ops.gated_scan(act.to(DEV), 0, H * D, 2 * H * D, 3 * H * D, meta, 1, state, out, H, D, V)
    else:
        ops.lightning_scan(act.to(DEV), 0, H * D, 3 * H * D, meta, 1, torch.tensor([0.9, 0.99], device=DEV), state, out, H, D, V,
                           torch.empty_like(act).to(DEV))
    infinite = torch.zeros(tokens, H * V, dtype=torch.bool)
    infinite[at:, column] = True
    assert torch.equal(torch.isinf(out.cpu()), infinite) and not torch.isnan(out).any()
    assert torch.isinf(state[0, 0, :, column]).all() and torch.isinf(state).sum() == D and not torch.isnan(state).any()


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("D,V", [(64, 128), (10, 40), (128, 40), (126, 30), (200, 128), (130, 30), (256, 16)])
def test_recurrence_does_not_show_its_columns_a_warp(D, V, gated):
    """More CTAs of sixteen columns than SMs (four columns a warp) against each entry alone (two) and token by token, in equal bits: key sizes
    of every number of elements a lane, with and without padding, 16-byte and single-element copies, columns that do not fill a CTA. The
    outputs of the longest entry lie within 2e-5 of the largest of the recurrence in 64 bits, the bound of the recurrence's other tests."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(D + V)
    lengths, H, E = [37, 1, 70, 16, 2, 33, 8, 9, 3, 5], 16, 10
    n, HD, HV = sum(lengths), 16 * D, 16 * V
    assert E * H * ((V + 15) // 16) > 148 >= H * ((V + 15) // 16)
    rows = [sum(lengths[:i]) for i in range(E)]
    x = torch.randn(n, 3 * HD + HV, generator=g) * 0.5
    x[:, HD:2 * HD] = torch.rand(n, HD, generator=g)
    x, decay = x.to(DEV), torch.linspace(0.5, 0.999, H, device=DEV)

    def run(first, count, entries, state):
        meta = torch.tensor([[e[k] for e in entries] for k in range(4)], dtype=torch.int32, device=DEV)
        part, out = x[first:first + count].contiguous(), torch.zeros(count, HV, device=DEV)
        if gated:
            ops.gated_scan(part, 0, HD, 2 * HD, 3 * HD, meta, len(entries), state, out, H, D, V)
        else:
            ops.lightning_scan(part, 0, 2 * HD, 3 * HD, meta, len(entries), decay, state, out, H, D, V, torch.empty_like(part))
        return out

    garbage = torch.randn(E, H, D, V, generator=g).to(DEV)
    together, alone, single = garbage.clone(), garbage.clone(), garbage.clone()
    whole = run(0, n, [(E - 1 - i, rows[i], lengths[i], 0) for i in range(E)], together)
    for i in range(E):
        assert torch.equal(run(rows[i], lengths[i], [(E - 1 - i, 0, lengths[i], 0)], alone), whole[rows[i]:rows[i] + lengths[i]])
        for t in range(lengths[i]):
            assert torch.equal(run(rows[i] + t, 1, [(E - 1 - i, 0, 1, t)], single)[0], whole[rows[i] + t])
    assert torch.equal(together, alone) and torch.equal(together, single)
    longest = x[rows[2]:rows[2] + lengths[2]].double()
    if not gated:
        longest = torch.nn.functional.silu(longest)
    q, f, k = (longest[:, i * HD:(i + 1) * HD].view(-1, H, D) for i in range(3))
    v, S, want = longest[:, 3 * HD:].view(-1, H, V), torch.zeros(H, D, V, dtype=torch.float64, device=DEV), []
    for t in range(lengths[2]):
        S = (f[t][:, :, None] if gated else decay.double()[:, None, None]) * S + k[t][:, :, None] * v[t][:, None, :]
        want.append(torch.einsum("hdv,hd->hv", S, q[t]).reshape(-1))
    want = torch.stack(want)
    assert (whole[rows[2]:rows[2] + lengths[2]].double() - want).abs().max() <= 2e-5 * float(want.abs().max())


@pytest.mark.parametrize("bw,B,n", [(128, 2, 330), (100, 3, 330), (33, 2, 1410), (16, 3, 330), (272, 1, 330), (1040, 1, 330)])
def test_gates_do_not_show_their_form(bw, B, n):
    """8 and 16 tokens a block, 16 and 32 tokens that share staged weights; sixteen bytes, four weights or one a request: the bits of a few
    tokens in those of n, with float32 weights and with the same numbers stored in bfloat16."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(bw)
    C = bw * B
    dev = lambda *s, k=0.3: (torch.randn(*s, generator=g) * k).to(DEV)
    proj, u, yb, rb, ib, lam = dev(2, n, 2 * C), dev(n, C), dev(C), dev(C), dev(C), dev(C) - 3.0
    gate_w = dev(B, bw, 2 * bw).bfloat16()

    def run(m, weights):
        outs = [torch.empty(m, C, device=DEV) for _ in range(3)]
        ops.rglru_gates(weights, rb, ib, lam, yb, u[:m].contiguous(), proj[:, :m].contiguous(), *outs)
        return outs

    whole = run(n, gate_w.float())
    for m in (1, 7, 8, 32, 33, 128, 129, 319, n):
        for weights in (gate_w, gate_w.float()):
            for x, w in zip(run(m, weights), whole):
                assert torch.equal(x, w[:m]), m


@pytest.mark.parametrize("C,K,P,n", [(2048, 4, 2, 300), (2048, 8, 1, 1030), (2048, 4, 9, 80), (2050, 4, 1, 80), (64, 16, 3, 5)])
def test_convolution_does_not_show_its_form(C, K, P, n):
    """One and four channels a thread, one and four rows, taps in registers or not: the bits of a few rows in those of n, and the rows within
    K + P roundings of the sum of the magnitudes in 64 bits."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(C + K)
    proj, xb, cb, taps = (torch.randn(*s, generator=g).to(DEV) for s in ((P, n, 2 * C), (C,), (C,), (C, K)))
    pos, slot = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)

    def run(m):
        u = torch.empty(m, C, device=DEV)
        ops.rglru_conv(proj[:, :m].contiguous(), xb, taps, cb, pos[:m], slot[:m], torch.full((1, K, C), 7.0, device=DEV), u)
        return u

    whole = run(n)
    for m in (1, 5, 33, 70, 256):
        if m < n:
            assert torch.equal(run(m), whole[:m]), m
    x = proj[:, :, C:].double().sum(0) + xb.double()
    x = torch.cat([torch.zeros(K - 1, C, dtype=torch.float64, device=DEV), x])
    want = sum(taps[:, j].double() * x[j:j + n] for j in range(K)) + cb.double()
    size = sum(taps[:, j].double().abs() * x[j:j + n].abs() for j in range(K)) + cb.double().abs() + P * 4.0
    assert ((whole.double() - want).abs() <= (K + P + 2) * 2.0 ** -23 * size * P).all()


@pytest.mark.parametrize("HD,HV", [(6, 10), (250, 130), (128, 64)])
def test_gates_of_linear_attention_do_not_show_the_rows(HD, HV):
    """Single elements, one and four a thread, and four neighbouring ones: the bits of a few rows in those of 1,030, and 64 bits within 2e-6."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(HD)
    n, dev = 1030, lambda *s: torch.randn(*s, generator=g).to(DEV)
    proj, fb, low = dev(3, n, 2 * HD + HV), dev(HD), torch.rand(HD, generator=g).to(DEV)

    def run(m):
        act = torch.empty(m, 3 * HD + HV, device=DEV)
        ops.hgrn2_activate(proj[:, :m].contiguous(), fb, low, act, HD, HV)
        return act

    whole = run(n)
    for m in (1, 1024, 1025):
        assert torch.equal(run(m), whole[:m])
    z = proj.double().sum(0)
    gate = low.double() + (1 - low.double()) * torch.sigmoid(z[:, HD:2 * HD] + fb.double())
    want = torch.cat([torch.nn.functional.silu(z[:, :HD]), gate, 1 - gate, z[:, 2 * HD:]], 1)
    assert (whole.double() - want).abs().max() <= 2e-6 * float(want.abs().max())      # a few roundings of sums of three


@pytest.mark.parametrize("H", [516, 1024, 2048, 2050, 3072, 4100, 9000])
def test_norms_do_not_show_the_rows(H):
    """As many rows as run at once, and more: other numbers of partial sums on their way and of blocks an SM, the same bits."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(H)
    n, w, b = 760, torch.randn(H, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV)
    h, parts = torch.randn(n, H, generator=g).to(DEV), torch.randn(9, n, H, generator=g).to(DEV)

    def run(m, norm):
        x, out = h[:m].clone(), torch.empty(m, H, device=DEV)
        if norm == "rms":
            ops.rmsnorm(x, w, 1e-5, out, partials=parts[:, :m].contiguous())
        else:
            ops.layernorm(x, w, b, 1e-5, out, partials=parts[:, :m].contiguous())
        return torch.cat([x, out], 1)

    for norm in ("rms", "layer"):
        whole = run(n, norm)
        for m in (1, 149, 297, 741):
            assert torch.equal(run(m, norm), whole[:m]), (norm, m)


@pytest.mark.parametrize("D,rot", [(64, 32), (96, 24), (64, 0), (64, 64)])
@pytest.mark.parametrize("P", [1, 2, 9])
def test_rotation_does_not_show_the_number_of_tokens(D, rot, P):
    """A pair a thread for a few tokens of heads rotated in part, four pairs otherwise: the bits of a few tokens in those of 70."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(D + rot)
    n, Hq, Hkv, page = 70, 5, 2, 16
    qkv = torch.randn(P, n, (Hq + 2 * Hkv) * D, generator=g).to(DEV)
    pos, slots = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    table, pages = torch.randn(n, max(rot // 2, 1), 2, generator=g).to(DEV), torch.arange(5, dtype=torch.int32, device=DEV)[None]

    def run(m):
        q, cache = torch.empty(m, Hq * D, device=DEV), torch.zeros(5, 2, Hkv, page, D, device=DEV)
        ops.rope_append(qkv[:, :m].contiguous(), pos[:m], slots[:m], table, rot, q, cache, pages, Hq, Hkv, D)
        return q, cache.permute(0, 3, 1, 2, 4).reshape(5 * page, -1)[:m]

    whole = run(n)
    for m in (1, 16, 17, 64, 65):
        for x, w in zip(run(m), whole):
            assert torch.equal(x, w[:m]), m


@pytest.mark.parametrize("W", [24, 2048, 4100])
def test_one_partial_buffer_gives_the_bits_of_several(W):
    """The forms for a single partial buffer against the same buffer beside a second one of zeros (x + 0 has the bits of x)."""
    from stride_b200.kernels import ops
    g = torch.Generator().manual_seed(W)
    n, dev = 9, lambda *s: torch.randn(*s, generator=g).to(DEV)
    two = lambda p: torch.cat([p, torch.zeros_like(p)])
    up, h, w, b, o = dev(1, n, W), dev(n, W), dev(W), dev(W), dev(n, W)

    def polynorm(p):
        out = torch.empty(n, W, device=DEV)
        ops.polynorm(p, out, (0.7, -0.3, 0.2, 0.05), 1e-5)
        return out

    def layernorm(p):
        x, out = h.clone(), torch.empty(n, W, device=DEV)
        ops.layernorm(x, w, b, 1e-5, out, partials=p)
        return torch.cat([x, out])

    def gated_norm(p):
        out = torch.empty(n, W, device=DEV)
        ops.gated_rmsnorm(o, p, 0, w, 1e-5, out)
        return out

    def hgrn2(p):
        out = torch.empty(n, 3 * (W // 4) + W // 2, device=DEV)
        ops.hgrn2_activate(p, w[:W // 4], torch.sigmoid(b[:W // 4]), out, W // 4, W // 2)
        return out

    def lightning(p):
        H = {24: 1, 2048: 4, 4100: 5}[W]
        D, V = W // 4 // H, W // 2 // H
        state, out, meta = torch.zeros(1, H, D, V, device=DEV), torch.empty(n, H * V, device=DEV), torch.tensor([[0], [0], [n], [0]], dtype=torch.int32, device=DEV)
        ops.lightning_scan(p, 0, H * D, 2 * H * D, meta, 1, torch.full((H,), 0.9, device=DEV), state, out, H, D, V, torch.empty(n * W, device=DEV))
        return torch.cat([out.flatten(), state.flatten()])

    def rope(p):
        D, Hq, Hkv = 8, W // 8 - 2, 1
        turn = torch.stack([torch.linspace(0, 2, 64).cos(), torch.linspace(0, 2, 64).sin()], -1).view(16, 4, 2).to(DEV)
        q, cache = torch.empty(n, Hq * D, device=DEV), torch.zeros(1, 2, Hkv, 16, D, device=DEV)
        ops.rope_append(p, torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV), turn, D, q, cache,
                        torch.zeros(1, 1, dtype=torch.int32, device=DEV), Hq, Hkv, D)
        return torch.cat([q.flatten(), cache.flatten()])

    for form in (polynorm, layernorm, gated_norm, hgrn2, lightning) + ((rope,) if W % 8 == 0 else ()):
        assert torch.equal(form(up), form(two(up))), form.__name__
