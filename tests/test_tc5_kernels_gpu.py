"""The tcgen05 kernels that stand beside mma.sync kernels of the same arithmetic: equal bits, and a plain computation in 64 bits."""
import subprocess
import sys
from ctypes import c_float, c_int, c_int64, c_void_p
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"
INF, NAN = float("inf"), float("nan")


def _call(name, argtypes, args):
    from stride_b200.kernels import ops
    lib, fn = ops._fn("masked_attention", name, argtypes)
    ops._check(lib, fn(*args))


def _kernels(call):
    """What call() returns and the names of the kernels that it launches."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        result = call()
        torch.cuda.synchronize()
    return result, " ".join(e.name for e in p.events())


def _latent_case(entries, H, G, page, odd=(), seed=0):
    """q, cache layer, block table, entry meta and sinks; entries are (tokens, tokens in front), memory that no token filled is NaN, `odd` are
    (entry, position, element, value) of latents."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    D, n = 512, sum(l for l, _ in entries)
    need = [-(-(l + f) // page) for l, f in entries]
    cache = torch.full((sum(need) + 2, 1, G, page, D), NAN, device=DEVICE, dtype=torch.bfloat16)
    order = torch.randperm(sum(need) + 2, generator=torch.Generator().manual_seed(seed)).tolist()
    table, meta, at, row = torch.zeros((len(entries), max(need)), dtype=torch.int32), [], 0, 0
    for e, (l, f) in enumerate(entries):
        table[e, :need[e]] = torch.tensor(order[at:at + need[e]], dtype=torch.int32)
        meta.append([e, row, l, f])
        at, row = at + need[e], row + l
    table = table.to(DEVICE)
    for e, (l, f) in enumerate(entries):
        j = torch.arange(l + f, device=DEVICE)
        for g in range(G):
            cache[table[e, j // page].long(), 0, g, j % page] = torch.randn((l + f, D), device=DEVICE, generator=gen).bfloat16()
    for e, j, c, v in odd:
        cache[table[e, j // page].long(), 0, 0, j % page, c] = v
    q = (torch.randn((n, H * D), device=DEVICE, generator=gen) * 0.5).bfloat16()
    return q, cache, table, torch.tensor(meta, dtype=torch.int32).T.contiguous().to(DEVICE), torch.randn(H, device=DEVICE, generator=gen)


def _latent(case, window, pages, longest=0):
    """pages: of the arena, or 0: the form that addresses pages by TMA is left out."""
    q, cache, table, meta, sinks = case
    H, G = sinks.numel(), cache.shape[2]
    out = torch.zeros_like(q)
    _call("sb_masked_attention_tiles",
          [c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_int64, c_int64, c_int64, c_void_p, c_int, c_int, c_void_p, c_void_p] +
          [c_int] * 8 + [c_float, c_int, c_int, c_float, c_void_p],
          [q.data_ptr(), out.data_ptr(), cache.data_ptr(), pages, longest, table.data_ptr(), table.shape[1], cache.shape[3], cache.stride(0), 0, cache.stride(2),
           meta.data_ptr(), meta.stride(0), meta.shape[1], None, sinks.data_ptr(), q.shape[0], H, G, 512, 512, 512, window, 0, 0.03, 0, 0, 0.0,
           torch.cuda.current_stream().cuda_stream])
    torch.cuda.synchronize()
    return out


LATENT = [  # entries, H, G, window, page size, odd latents
    ([(16, 0)], 16, 1, 0, 64, ()), ([(17, 47)], 16, 1, 0, 64, ()), ([(1, 700), (1, 63), (1, 64), (3, 0)], 16, 1, 100, 64, ()), ([(1, 200)], 64, 1, 0, 16, ()), ([(64, 0)], 16, 1, 0, 64, ()),
    ([(200, 0), (33, 100), (65, 7)], 16, 1, 1024, 64, ()), ([(150, 100), (90, 7)], 16, 1, 70, 16, ()), ([(70, 300)], 16, 1, 3, 8, ()), ([(170, 300)], 16, 1, 3, 8, ()),
    ([(100, 500), (41, 7)], 32, 2, 64, 128, ()), ([(100, 30)], 4, 1, 65, 32, ()), ([(20, 50)], 128, 1, 0, 64, ()), ([(300, 0)], 1, 1, 0, 64, ()),
    # as many tiles as entries of that many tokens can have: a token beyond every entry's last full tile
    ([(9, 130), (17, 0), (1, 5), (25, 40)], 16, 1, 0, 64, ()), ([(3, 200)] * 5, 64, 1, 0, 64, ()), ([(1, 127)] * 55, 128, 1, 0, 64, ()),
    ([(17, 150), (17, 20)], 16, 2, 0, 64, ()),
    # infinities and NaN at keys that some rows of a tile see and others do not: at the causal edge and at the window's
    ([(100, 0), (64, 3)], 16, 1, 0, 64, ((0, 50, 3, INF), (0, 51, 300, NAN), (1, 66, 511, -INF))),
    ([(100, 30), (64, 3)], 16, 1, 20, 64, ((0, 50, 3, INF), (0, 129, 300, NAN), (1, 3, 511, -INF), (1, 4, 0, INF))),
]


@pytest.mark.parametrize("entries, H, G, window, page, odd", LATENT)
def test_latent_attention_on_tcgen05_has_the_bits_of_the_tile_kernel(entries, H, G, window, page, odd):
    from stride_b200.kernels import ops
    word = ops.shared_status_word({"masked_attention"})
    case = _latent_case(entries, H, G, page, odd)
    many, names = _kernels(lambda: _latent(case, window, case[1].shape[0], max(l + f for l, f in entries)))
    assert ("latent_attention_tc5_kernel" in names) == (entries != [(70, 300)])       # (a window of three over pages of eight, few blocks)
    assert torch.equal(many.view(torch.int16), _latent(case, window, 0).view(torch.int16))
    assert word.item() == 0
    if odd:
        return
    # a plain computation in 64 bits. bfloat16 results have eight significant bits: half a unit in the last place is up to 2^-8 of the largest
    # element (2^-8 2^e beside a value of at least 2^e); scores and sums are of 32 bits
    q, cache, table, meta, sinks = case
    for e, row, l, f in meta.T.tolist():
        j = torch.arange(l + f, device=DEVICE)
        keys = torch.stack([cache[table[e, j // page].long(), 0, g, j % page] for g in range(G)]).double()
        s = torch.einsum("tgrd,gsd->grts", q[row:row + l].view(l, G, H // G, 512).double(), keys) * 0.03
        pos = torch.arange(f, f + l, device=DEVICE)[:, None]
        seen = (j[None, :] <= pos) & ((pos - j[None, :] < window) if window else True)
        s = torch.cat([s.masked_fill(~seen, -INF), sinks.double().view(G, H // G, 1, 1).expand(-1, -1, l, 1)], dim=-1)
        want = torch.einsum("grts,gsd->tgrd", torch.softmax(s, -1)[..., :-1], keys).reshape(l, -1)
        got = many[row:row + l].double()
        assert ((got - want).abs().max() / want.abs().max()).item() < 2.0 ** -8 + 1e-4


@pytest.mark.parametrize("count, length, H, G, window, longest, page, taken", [
    (55, 1, 16, 1, 0, 150, 64, True), (56, 1, 16, 1, 0, 150, 64, False), (37, 1, 16, 1, 0, 0, 64, True), (38, 1, 16, 1, 0, 127, 64, False),
    (38, 1, 16, 1, 0, 128, 64, True), (38, 1, 16, 1, 100, 700, 64, False), (55, 1, 32, 1, 0, 0, 64, True), (56, 1, 32, 1, 0, 0, 64, False),
    (8, 1, 4, 1, 0, 60, 64, False), (8, 1, 4, 1, 0, 128, 64, True), (1, 1, 1, 1, 0, 0, 64, False), (27, 1, 32, 2, 0, 128, 64, True),
    (28, 1, 32, 2, 0, 128, 64, False),
    # two tiles of rows an entry: one head a latent, four, and blocks of 16 rows around the SMs
    (1, 256, 1, 1, 100, 700, 64, False), (1, 256, 1, 1, 0, 276, 64, True), (1, 64, 4, 1, 16, 84, 64, True), (8, 256, 1, 1, 16, 276, 64, False),
    (10, 256, 1, 1, 16, 276, 64, True),
    # pages of eight
    (8, 1, 16, 1, 0, 60, 8, False), (8, 1, 16, 1, 0, 128, 8, True), (8, 1, 4, 1, 0, 128, 8, False), (2, 64, 16, 1, 0, 84, 8, False),
    (3, 64, 16, 1, 0, 84, 8, True), (8, 1, 16, 1, 0, 60, 16, True)])
def test_which_latent_attention_is_taken(count, length, H, G, window, longest, page, taken):
    """Both sides of the lines between the two forms, which have the same bits."""
    case = _latent_case([(length, 20)] * count, H, G, page)
    got, names = _kernels(lambda: _latent(case, window, case[1].shape[0], longest))
    assert ("latent_attention_tc5_kernel" in names) == taken
    assert torch.equal(got.view(torch.int16), _latent(case, window, 0).view(torch.int16))


HEADS = [  # n, H, K, N, partial sums of the gate, elements behind a row, elements behind a gate's row, whether the tcgen05 form is taken
    (130, 2, 128, 512, 0, 0, 64, False), (256, 1, 64, 64, 0, 0, 64, False), (127, 16, 192, 320, 0, 0, 64, False), (128, 1, 192, 64, 0, 0, 64, True),
    (300, 5, 192, 320, 0, 0, 64, True), (700, 4, 256, 64, 0, 8, 64, True), (383, 3, 512, 192, 0, 8, 64, True),
    # at the line of three quarters of the SMs (blocks of 64 x 64), and at one CTA of 64 columns an SM, where the columns become more
    (256, 27, 64, 64, 0, 0, 64, False), (256, 28, 64, 64, 0, 0, 64, True), (256, 37, 64, 128, 0, 0, 64, True), (256, 38, 64, 128, 0, 0, 64, True),
    (513, 15, 128, 256, 0, 0, 64, True), (2000, 5, 1024, 192, 0, 0, 64, True),
    # gates: several partial sums, few CTAs, too few tokens, widths and places without 16-byte accesses; then the form itself, in one round and in several
    (513, 2, 512, 128, 3, 0, 64, False), (257, 16, 512, 128, 9, 0, 64, False), (513, 2, 512, 128, 1, 0, 64, False), (511, 32, 512, 128, 1, 0, 64, False),
    (640, 16, 512, 128, 1, 0, 62, False), (640, 16, 512, 128, 1, 0, 65, False),
    (640, 16, 512, 128, 1, 0, 64, True), (512, 32, 512, 128, 1, 8, 4, True), (515, 16, 1024, 64, 1, 0, 64, True), (700, 30, 192, 128, 1, 0, 64, True),
    (700, 32, 512, 192, 1, 0, 64, True), (515, 16, 512, 320, 1, 0, 64, True), (1030, 18, 384, 256, 1, 0, 64, False), (1030, 24, 384, 256, 1, 0, 64, True), (2047, 32, 320, 64, 1, 0, 64, True),
    (2047, 32, 256, 64, 1, 0, 64, False),
]


@pytest.mark.parametrize("n, H, K, N, partials, pad, gate_pad, many", HEADS)
def test_matrix_per_head_has_one_result_for_any_number_of_rows(n, H, K, N, partials, pad, gate_pad, many):
    """The tcgen05 kernel where the rule says so, the mma.sync kernel for a few rows: the same bits, and nothing written beyond the rows or the
    columns."""
    gen = torch.Generator(device=DEVICE).manual_seed(n)
    x = torch.randn((n, H, K + pad), device=DEVICE, generator=gen).bfloat16()
    w = (torch.randn((H, K, N), device=DEVICE, generator=gen) * 0.05).bfloat16()
    width = H * N + gate_pad
    gate = torch.randn((partials, n, width), device=DEVICE, generator=gen) if partials else None

    def run(first, rows):
        out = torch.full((rows + 1, H, N + pad), 7.0, device=DEVICE, dtype=torch.bfloat16)
        at = gate.data_ptr() + 4 * first * width if partials else None
        _call("sb_head_linear_gated",
              [c_void_p, c_int64, c_int64, c_void_p, c_void_p, c_int64, c_int64] + [c_int] * 6 + [c_void_p, c_int, c_int64, c_int, c_void_p],
              [x[first:].data_ptr(), x.stride(0), x.stride(1), w.data_ptr(), out.data_ptr(), out.stride(0), out.stride(1), 1, rows, H, K, N, 0, at, partials,
               n * width, width, torch.cuda.current_stream().cuda_stream])
        torch.cuda.synchronize()
        assert (out[rows] == 7).all() and (out[:, :, N:] == 7).all()
        return out[:rows, :, :N]
    whole, names = _kernels(lambda: run(0, n))
    assert ("head_linear_tc5_kernel" in names) == many and ("head_linear_tc_kernel" in names) != many
    assert torch.equal(whole, torch.cat([run(a, min(60, n - a)) for a in range(0, n, 60)]))
    want = torch.einsum("nhk,hkm->nhm", x[..., :K].double(), w.double())
    if partials:
        want = want * torch.sigmoid(gate[..., :H * N].double().sum(0)).view(n, H, N)
    # half a unit in the last place of a bfloat16 (up to 2^-8 of the largest element) and sums of 32 bits whose terms the tensor cores truncate
    assert ((whole.double() - want).abs().max() / want.abs().max()).item() < 2.0 ** -8 + 1e-4


@pytest.mark.parametrize("n", [129, 145, 256, 300, 513, 700])
@pytest.mark.parametrize("M, K, gated", [(1040, 520, False), (1042, 520, False), (300, 2048, False), (1040, 264, True), (1032, 264, True), (1034, 264, True)])
def test_products_of_many_tokens_store_what_products_of_a_few_store(n, M, K, gated):
    """More than 128 tokens: tiles that go to memory by TMA (rows of a multiple of four elements) or element by element, and the SwiGLU epilogue
    of pairs with 16-byte stores (a multiple of eight features) or without; portions of at most 100 tokens take neither. The same bits."""
    from stride_b200.kernels import ops
    gen = torch.Generator(device=DEVICE).manual_seed(n)
    x = torch.randn((n, K), device=DEVICE, generator=gen).bfloat16()
    w = (torch.randn((M, K), device=DEVICE, generator=gen) * 0.05).bfloat16()
    S = 1 if gated else ops.gemm_tc_splits(M, K)

    def run(part):
        rows = part.shape[0]
        if gated:
            out = torch.full((rows + 1, M // 2), 7.0, device=DEVICE, dtype=torch.bfloat16)
            ops.gemm_tc(part, w, out[:rows], ops.SWIGLU, half_rows=M // 2)
            assert (out[rows] == 7).all()
            return out[:rows]
        ranges = S if rows <= ops.gemm_tc_partial_tokens() else 1
        out = torch.full((ranges * rows + 1, M), 7.0, device=DEVICE)
        ops.gemm_tc(part, w, out[:-1].view(ranges, rows, M) if ranges > 1 else out[:-1], ops.STORE, splits=S)
        assert (out[-1] == 7).all()
        total = out[:rows].clone()
        for s in range(1, ranges):
            total += out[s * rows:(s + 1) * rows]
        return total
    whole = run(x)
    assert torch.equal(whole, torch.cat([run(x[a:a + 100]) for a in range(0, n, 100)]))
    y = x.double() @ w.double().T
    if gated:
        y = torch.nn.functional.silu(y[:, :M // 2]) * y[:, M // 2:]
    # bfloat16 results: half a unit in the last place, 2^-8 of the largest; sums of 32 bits whose terms the tensor cores truncate (2e-6 on average
    # over 2,048 of them)
    assert ((whole.double() - y).abs().max() / y.abs().max()).item() < (2.0 ** -8 + 1e-4 if gated else 1e-4)
    assert ops.gemm_tc_status() == 0


@pytest.mark.parametrize("n", [2048, 2061])
@pytest.mark.parametrize("M, K", [(3072, 136), (5124, 136), (3072, 2048), (5124, 2048), (5122, 136)])
def test_pairs_that_walk_several_tiles_store_what_products_of_a_few_store(M, K, n):
    """96 to 189 tiles on 74 pairs of CTAs: a pair's last tile goes to memory by TMA over the ring, the ones in front of it element by element;
    one and several ranges of K, rows that the tiles do not divide, and rows that TMA does not take."""
    test_products_of_many_tokens_store_what_products_of_a_few_store(n, M, K, False)


@pytest.mark.parametrize("K", [3064, 3072, 3080])
@pytest.mark.parametrize("M, n", [(8192, 700), (8204, 513), (16384, 300)])
def test_gated_products_that_take_as_many_rounds_on_pairs(M, n, K):
    """As many rounds on pairs of CTAs as with two weight tiles a CTA: K at the line between the two, features that no tile and no 16-byte store divides."""
    test_products_of_many_tokens_store_what_products_of_a_few_store(n, M, K, True)


FIRST_CALL = """
import torch
from stride_b200.kernels import ops
x = torch.randn((300, 16, 128), device="cuda").bfloat16()
w = torch.randn((16, 128, 512), device="cuda").bfloat16()
few, many = (torch.zeros((n, 16, 512), device="cuda", dtype=torch.bfloat16) for n in (60, 300))
ops.head_linear(x[:60], w, few)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    ops.head_linear(x, w, many)
graph.replay()
torch.cuda.synchronize()
assert torch.equal(few, many[:60])
"""


def test_a_first_call_on_many_rows_can_be_captured():
    """A program that has only run a few rows may record many: the kernel's status word is there without an allocation."""
    run = subprocess.run([sys.executable, "-c", FIRST_CALL], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
