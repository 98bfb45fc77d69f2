"""The float32 path's product and attention at the sizes where their rules change hands: few rows and tiles of rows, one
chunk of k and many, one group of chunks and eight, a row's keys in one span and in eight, spans side by side and one
after the other. Every result against 64-bit arithmetic within a bound from the order of the sums, and the same bits
whoever computes it."""

import os
import subprocess
import sys

import pytest
import torch

from test_kernels_gpu import Meta, fill_cache, make_cache

pytestmark = pytest.mark.gpu


def cuda():
    from fusezap_core_b200.kernels import cuda_ops
    return cuda_ops("float32")


@pytest.mark.parametrize("N,K", [(1, 1), (9, 33), (96, 31), (130, 1024), (64, 1028), (4097, 136), (200, 2050), (896, 4864), (16385, 256)])
def test_linear(N, K):
    cu = cuda()
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randn(200, K, generator=g, device="cuda")
    w = torch.randn(N, K, generator=g, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda")
    exact = a.double() @ w.double().T + bias.double()
    # a chain of K / 32 (rounded up to a multiple of 32) fmaf, at most 32 + 8 additions and the bias, each rounding by
    # 2^-24 of a partial sum that is at most the sum of magnitudes
    steps = 32 * -(-K // 1024) + 41
    bound = steps * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs().double())
    full = torch.empty(200, N, device="cuda")
    cu.linear(a, w, bias, full)
    assert bool(((full.double() - exact).abs() <= bound).all())
    for rows in (1, 2, 3, 5, 8, 9, 16, 17, 32, 33, 64, 65, 129):
        part = torch.full((rows + 1, N), float("nan"), device="cuda")
        cu.linear(a[7:7 + rows].contiguous(), w, bias, part[:rows])
        assert torch.equal(part[:rows], full[7:7 + rows]), f"{rows} rows"
        assert bool(part[rows].isnan().all()), f"{rows} rows: written beyond the last"
    # operands off the 16-byte boundaries: read one by one, the same bits
    off_a, off_w = torch.empty(5 * K + 1, device="cuda")[1:].view(5, K), torch.empty(N * K + 1, device="cuda")[1:].view(N, K)
    off_a.copy_(a[:5])
    off_w.copy_(w)
    part = torch.empty(5, N, device="cuda")
    cu.linear(off_a, off_w, bias, part)
    assert torch.equal(part, full[:5])
    # an infinity stays in its own row and column
    bad = a[:20].clone()
    bad[3, K // 2] = float("inf")
    out = torch.empty(20, N, device="cuda")
    cu.linear(bad, w, bias, out)
    assert torch.equal(out[:3], full[:3]) and torch.equal(out[4:], full[4:20]) and not bool(out[3].isfinite().any())


@pytest.mark.parametrize("dtype,N,K", [("float32", 16385, 1028), ("float32", 16385, 1030), ("float32", 9500, 33), ("float32", 384, 96),
                                       ("bfloat16", 9500, 33), ("bfloat16", 9500, 1030), ("bfloat16", 384, 97), ("bfloat16", 100, 17)])
def test_linear_bits_in_every_kernel(dtype, N, K):
    """The bits of few rows from tiles of 32 and of 64 rows and from the wide tiles, with K off whole stages, chunks longer
    than 32 and operands that are read one by one, misaligned ones among them."""
    from fusezap_core_b200.kernels import cuda_ops
    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    cu = cuda_ops(dtype)
    g = torch.Generator(device="cuda").manual_seed(N + K)
    rows = 400
    a = torch.randn(rows, K, generator=g, device="cuda").to(dt)
    w = torch.randn(N, K, generator=g, device="cuda").to(dt)
    few = torch.empty(rows, N, device="cuda")
    for r in range(0, rows, 16):
        cu.linear(a[r:r + 16].contiguous(), w, None, few[r:r + 16])
    steps = 32 * -(-K // 1024) + 41      # (as above)
    bound = steps * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T)
    assert bool(((few.double() - a.double() @ w.double().T).abs() <= bound).all())
    for m in (33, 64, 200, 400):
        out = torch.full((m + 1, N), float("nan"), device="cuda")
        cu.linear(a[:m].contiguous(), w, None, out[:m])
        assert torch.equal(out[:m], few[:m]) and bool(out[m].isnan().all()), f"{m} rows"
    off_a, off_w = torch.empty(200 * K + 1, dtype=dt, device="cuda")[1:].view(200, K), torch.empty(N * K + 1, dtype=dt, device="cuda")[1:].view(N, K)
    off_a.copy_(a[:200])
    off_w.copy_(w)
    out = torch.empty(200, N, device="cuda")
    cu.linear(off_a, off_w, None, out)
    assert torch.equal(out, few[:200])


def test_linear_from_two_threads():
    """Products whose blocks need different amounts of shared memory, first called by two threads at once in a process that
    has launched none of them (the limit of a kernel's shared memory is set at its first call)."""
    code = """
import threading, torch
from fusezap_core_b200.kernels.table import CudaOps
from test_float32_kernels_gpu import thread_sizes
torch.zeros(1, device="cuda")
meet, bad = threading.Barrier(2), []
def work(order):
    ops = CudaOps("float32", "cuda:0")
    with torch.cuda.stream(torch.cuda.Stream()):
        for m, n, k in order:
            a, w, out = torch.ones(m, k, device="cuda"), torch.ones(n, k, device="cuda"), torch.empty(m, n, device="cuda")
            meet.wait(60)
            ops.linear(a, w, None, out)
            if not bool((out == k).all()): bad.append((m, n, k))
def guarded(order):
    try: work(order)
    except BaseException as e:
        bad.append(repr(e)); meet.abort()
sizes = thread_sizes()
threads = [threading.Thread(target=guarded, args=(o,)) for o in (sizes, sizes[::-1])]
for t in threads: t.start()
for t in threads: t.join()
assert not bad, bad
"""
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(p for p in sys.path if p))
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300)


def test_attention_and_bfloat16_products_from_two_threads():
    """The same of the 32-bit attention's kernels, whose blocks need more or less by head size, heads and rows, and of the
    tensor-core products, whose rings are as deep as K asks for."""
    code = """
import threading, torch
from fusezap_core_b200.kernels.table import CudaOps
from test_float32_kernels_gpu import thread_calls
torch.zeros(1, device="cuda")
meet, bad = threading.Barrier(2), []
def work(order):
    ops = {t: CudaOps(t, "cuda:0") for t in ("float32", "bfloat16")}
    with torch.cuda.stream(torch.cuda.Stream()):
        for call, args in order:
            meet.wait(60)
            if not call(ops, *args): bad.append((call.__name__, args))
def guarded(order):
    try: work(order)
    except BaseException as e:
        bad.append(repr(e)); meet.abort()
calls = thread_calls()
threads = [threading.Thread(target=guarded, args=(o,)) for o in (calls, calls[::-1])]
for t in threads: t.start()
for t in threads: t.join()
assert not bad, bad
"""
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(p for p in sys.path if p))
    subprocess.run([sys.executable, "-c", code], check=True, env=env, timeout=300)


def thread_calls():
    def product(ops, m, n, k):
        a, w = (torch.ones(r, k, dtype=torch.bfloat16, device="cuda") for r in (m, n))
        out = torch.empty(m, n, dtype=torch.float32, device="cuda")
        ops["bfloat16"].linear(a, w, None, out)
        return bool((out == k).all())

    def attention(ops, rows, heads, hd):
        cache = make_cache(20, heads, 16, hd, torch.float32, "cuda")
        cache.pool.fill_(1.0)
        q = torch.ones(rows, 2 * heads * hd, device="cuda")
        out = torch.empty_like(q)
        ops["float32"].paged_attention(q, cache, Meta(list(range(300 - rows, 300)), [0] * rows, [list(range(20))], "cuda"), out,
                                       2 * heads, heads, hd, hd ** -0.5, 0)
        return bool(((out - 1.0).abs() < 1e-5).all())

    return [(product, (m, n, k)) for m in (1, 20, 40, 100, 200) for n, k in ((256, 128), (896, 896), (896, 4864), (9728, 896))] \
        + [(attention, (rows, heads, hd)) for rows in (1, 40, 300) for heads in (1, 4) for hd in (40, 48, 56, 64, 72, 96, 128, 160, 256)]


def thread_sizes():
    return [(m, n, k) for m in (1, 3, 8, 16, 32, 64) for n, k in ((64, 64), (896, 896), (896, 4864), (9728, 896))]


@pytest.mark.parametrize("Hq,Hkv,hd,bs,window", [(14, 2, 64, 16, 0), (3, 1, 32, 4, 0), (8, 8, 128, 8, 0), (40, 1, 48, 16, 0), (4, 2, 64, 16, 300),
                                                 (2, 1, 512, 16, 0), (6, 2, 256, 1, 77), (2, 2, 20, 16, 0)])
def test_attention_bits_do_not_depend_on_who_computes_them(Hq, Hkv, hd, bs, window):
    cu = cuda()
    lengths = [1100, 129, 31]
    mb = -(-max(lengths) // bs)
    g = torch.Generator().manual_seed(hd + window)
    perm = torch.randperm(3 * mb + 2, generator=g).tolist()
    table = [perm[r * mb:(r + 1) * mb] for r in range(3)]
    cp = make_cache(3 * mb + 2, Hkv, bs, hd, torch.float32, "cpu")
    fill_cache(cp, table, lengths, g)
    cc = make_cache(3 * mb + 2, Hkv, bs, hd, torch.float32, "cuda")
    cc.pool.copy_(cp.pool)
    # a portion that ends at the longest context, one that starts a request, single tokens, a padding row
    rows = [(0, p) for p in range(800, 1100)] + [(2, p) for p in range(31)] + [(-1, 0)] + [(1, 128), (0, 127), (0, 128)]
    q = torch.randn(len(rows), Hq * hd, generator=g).cuda()
    many = torch.full((len(rows), Hq * hd), float("nan"), device="cuda")
    scale = hd ** -0.5

    def attend(index, out, cache=cc):
        cu.paged_attention(q[index].contiguous(), cache, Meta([rows[i][1] for i in index], [rows[i][0] for i in index], table, "cuda"), out,
                           Hq, Hkv, hd, scale, window)

    attend(list(range(len(rows))), many)
    assert bool(many.isfinite().all()) and float(many[331].abs().max()) == 0.0
    for index in ([0], [150], [299], [300], [330], [332], [333], [334], [299, 332, 331, 334], list(range(290, 335)), list(range(100, 300))):
        few = torch.full((len(index), Hq * hd), float("nan"), device="cuda")
        attend(index, few)
        assert torch.equal(few, many[index]), f"rows {index[:4]}"
    # against 64 bits: scores off by (hd + 2) roundings of at most sum |q||k| * scale, weights by that and an exponential,
    # sums by the chunk, span and merge roundings (fewer than 200 for 1,100 keys) of values of at most max |v|
    for i in (0, 299, 330, 332, 333):
        r, p = rows[i]
        lo = max(0, p - window + 1) if window else 0
        at = torch.tensor([table[r][k // bs] for k in range(lo, p + 1)]), torch.tensor([k % bs for k in range(lo, p + 1)])
        keys, values = (cp.pool[at[0], j][torch.arange(p + 1 - lo), :, at[1]].double() for j in (0, 1))      # (keys, Hkv, hd)
        qi = q[i].cpu().double().view(Hkv, Hq // Hkv, hd)
        s = torch.einsum("hgd,khd->hgk", qi, keys) * scale
        ref = torch.einsum("hgk,khd->hgd", s.softmax(-1), values).reshape(-1)
        s_err = (hd + 2) * 2.0 ** -24 * float(torch.einsum("hgd,khd->hgk", qi.abs(), keys.abs()).max()) * scale
        bound = (2 * s_err + 210 * 2.0 ** -24) * float(values.abs().max())
        assert float((many[i].cpu().double() - ref).abs().max()) <= bound
    # keys and values that a row does not see yet take no part, whatever they hold
    spoiled = make_cache(3 * mb + 2, Hkv, bs, hd, torch.float32, "cuda")
    spoiled.pool.copy_(cp.pool)
    for k in range(850, 1100):
        spoiled.pool[table[0][k // bs], :, :, k % bs] = float("inf") if k % 2 else float("nan")
    for index in ([0, 20, 49], list(range(0, 50)), [333, 334]):
        few = torch.empty(len(index), Hq * hd, device="cuda")
        attend(index, few, spoiled)
        assert torch.equal(few, many[index])
    whole = torch.empty(len(rows), Hq * hd, device="cuda")
    attend(list(range(len(rows))), whole, spoiled)
    assert torch.equal(whole[:50], many[:50]) and torch.equal(whole[300:], many[300:])
    cu.check_errors()


def test_attention_with_more_heads_and_slices_than_a_grid_is_high():
    """33,000 kv heads of nine query heads at a head size where a block takes eight: two slices of each kv head, 66,000 in
    all, more than the 65,535 blocks that a grid's second dimension holds."""
    from fusezap_core_b200.kernels import cuda_ops
    cu = cuda_ops("bfloat16")
    Hkv, G, hd, bs = 33000, 9, 264, 4
    g = torch.Generator(device="cuda").manual_seed(1)
    cache = make_cache(1, Hkv, bs, hd, torch.bfloat16, "cuda")
    cache.pool.normal_(generator=g)
    q = torch.randn(2, Hkv * G * hd, generator=g, device="cuda").bfloat16()
    out = torch.empty_like(q)
    cu.paged_attention(q, cache, Meta([0, 2], [0, 0], [[0]], "cuda"), out, Hkv * G, Hkv, hd, hd ** -0.5, 0)
    cu.check_errors()
    # the first row sees one key, whose value it returns; the second one's softmax has three
    assert torch.equal(out[0].view(Hkv, G, hd), cache.values[0, :, 0][:, None].expand(Hkv, G, hd))
    s = torch.einsum("hgd,hkd->hgk", q[1].view(Hkv, G, hd).float(), cache.keys[0, :, :3].float()) * hd ** -0.5
    ref = torch.einsum("hgk,hkd->hgd", s.softmax(-1), cache.values[0, :, :3].float())
    # half a bfloat16 step of the result, and the 32-bit sums
    assert bool(((out[1].view(Hkv, G, hd).float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all())


def test_rows_of_different_requests_do_not_wait_for_each_other():
    """Blocks hold several rows only where these can be of one portion."""
    rows = cuda().core.fz_attn_simt_rows
    # decoded tokens: a row's spans side by side while rows are few, then a row per block
    assert [rows(n, 14, 2, 64, 300, 1) for n in (1, 64, 100, 300, 4000)] == [0, 0, 1, 1, 1]
    assert [rows(n, 14, 2, 64, 2048, 1) for n in (1, 148, 300, 4000)] == [0, 0, 1, 1]
    # portions: rows share keys, as many as they have and as leave blocks for every SM
    assert [rows(n, 14, 2, 64, n, n) for n in (400, 2000)] == [2, 4]
    assert rows(4000, 14, 2, 64, 300, 3) == 3 and rows(300, 8, 8, 64, 300, 300) == 8


@pytest.mark.parametrize("dtype,Hq,Hkv,hd,bs,window", [("float32", 4, 4, 32, 16, 0), ("float32", 6, 2, 64, 8, 40), ("bfloat16", 3, 1, 48, 16, 0),
                                                       ("bfloat16", 8, 8, 80, 8, 33), ("bfloat16", 4, 2, 36, 16, 0), ("bfloat16", 40, 1, 24, 16, 0)])
def test_attention_rows_in_blocks(dtype, Hq, Hkv, hd, bs, window):
    """Runs of rows that start and end off the multiples of eight at which blocks change hands, runs of two requests whose
    positions continue, the same request at other positions, the same row twice, padding: every row has the bits that it
    has alone, whatever the longest run is said to be, and is right."""
    from fusezap_core_b200.kernels import cuda_ops
    from plain_ops import PlainOps
    dt = torch.float32 if dtype == "float32" else torch.bfloat16
    cu, pl = cuda_ops(dtype), PlainOps(dt)
    lengths = [700, 400, 90]
    mb = -(-700 // bs)
    g = torch.Generator().manual_seed(hd)
    perm = torch.randperm(3 * mb, generator=g).tolist()
    table = [perm[r * mb:(r + 1) * mb] for r in range(3)]
    cp = make_cache(3 * mb, Hkv, bs, hd, dt, "cpu")
    fill_cache(cp, table, lengths, g)
    cc = make_cache(3 * mb, Hkv, bs, hd, dt, "cuda")
    cc.pool.copy_(cp.pool)
    rows = [(2, 5)] + [(0, p) for p in range(301, 330)] + [(1, p) for p in range(330, 347)] + [(-1, 0)] * 2 + [(0, p) for p in range(673, 700)] \
        + [(0, 699), (0, 31), (0, 0), (1, 399)] + [(2, p) for p in range(60, 90)]
    q = torch.randn(len(rows), Hq * hd, generator=g).to(dt)

    def attend(index, longest):
        out = torch.full((len(index), Hq * hd), float("nan"), dtype=dt, device="cuda")
        meta = Meta([rows[i][1] for i in index], [rows[i][0] for i in index], table, "cuda")
        meta.max_portion = longest
        cu.paged_attention(q[index].cuda(), cc, meta, out, Hq, Hkv, hd, hd ** -0.5, window)
        return out

    every = list(range(len(rows))) * (6 if Hkv == 1 else 3)      # (enough rows for blocks of several)
    full = attend(every, 30)
    assert torch.equal(full, full[:len(rows)].repeat(len(every) // len(rows), 1))
    for longest in (1, 2, 3, 5, 1000):
        assert torch.equal(attend(every, longest), full), f"longest run {longest}"
    for i in (0, 1, 2, 3, 11, 29, 30, 46, 47, 50, 75, 76, 77, 78, 79, 80, len(rows) - 1):
        assert torch.equal(attend([i], 1)[0], full[i]), f"row {i}"
    ref = torch.empty(len(rows), Hq * hd, dtype=dt)
    pl.paged_attention(q, cp, Meta([p for _, p in rows], [r for r, _ in rows], table, "cpu"), ref, Hq, Hkv, hd, hd ** -0.5, window)
    # float32: 700 keys' sums in two orders; bfloat16: the roundings of the two results
    assert float((full[:len(rows)].float().cpu() - ref.float()).abs().max()) <= (1e-5 if dtype == "float32" else 2.0 ** -7) * float(ref.float().abs().max())
    cu.check_errors()
