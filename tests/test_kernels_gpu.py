"""Each CUDA kernel alone against the plain implementation's function for the same op, at sizes the
tiny models do not use: widths and vocabularies that are no power of two, head sizes in steps
of 16, odd numbers of heads and groups, scattered pages."""
import numpy as np
import pytest
import torch

import plain_qwen3 as plain
from conftest import rel_err

pytestmark = pytest.mark.gpu

DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
TOL = {"float32": 2e-5, "bfloat16": 1.2e-2}   # one kernel: a few float32 roundings, or one bfloat16 rounding of the output


def dev(a, dtype=torch.float32):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda").to(dtype)


def host(t):
    return t.float().cpu().numpy()


def as_stored(a, dtype):
    """What the kernel sees: the values after rounding to the storage dtype."""
    return plain.round_bf16(a.astype(np.float32)) if dtype == "bfloat16" else a.astype(np.float32)


@pytest.fixture(scope="module")
def ops():
    from tiny_inference_engine_b200 import ops
    return ops


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_embed(ops, dtype):
    """Widths that let a thread move 16 bytes of the table at a time, and one that does not."""
    rng = np.random.default_rng(0)
    for width in (72, 75, 4096):
        table = as_stored(rng.standard_normal((311, width)), dtype)
        ids = rng.integers(0, 311, 37)
        out = torch.full((37, width), float("nan"), device="cuda")
        ops.embed(dev(table, DT[dtype]), dev(ids, torch.int32), out)
        assert np.array_equal(host(out), plain.embed(table, ids).astype(np.float32))


def test_scatter_ids(ops):
    """tokens[dst[i]] = ids[src[i]] for the first n pairs; everything else is left as it is."""
    rng = np.random.default_rng(5)
    tokens = rng.integers(0, 1000, 700).astype(np.int32)
    ids = rng.integers(0, 1000, 300).astype(np.int32)
    dst = rng.permutation(700)[:300].astype(np.int32)
    src = rng.integers(0, 300, 300).astype(np.int32)
    for n in (0, 1, 129, 300):
        t = dev(tokens, torch.int32)
        ops.scatter_ids(t, dev(dst, torch.int32), dev(src, torch.int32), dev(ids, torch.int32), n)
        want = tokens.copy()
        want[dst[:n]] = ids[src[:n]]
        assert np.array_equal(host(t), want)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("dim", [72, 1000, 5120])
def test_add_rmsnorm(ops, dtype, dim):
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((9, dim)).astype(np.float32) * 3
    delta = as_stored(rng.standard_normal((9, dim)), dtype)
    w = (1 + 0.1 * rng.standard_normal(dim)).astype(np.float32)
    xd, out = dev(x), torch.empty(9, dim, device="cuda", dtype=DT[dtype])
    ops.add_rmsnorm(xd, dev(delta, DT[dtype]), dev(w), 1e-5, out)
    want_x = x.astype(np.float64) + delta
    assert np.abs(host(xd) - want_x).max() < 1e-6 * np.abs(want_x).max()        # the residual sum is float32
    assert rel_err(host(out), plain.rms_norm(want_x, w, 1e-5)) < TOL[dtype]
    # without a delta x is untouched; with rows only those rows come out and x is not written
    x2 = dev(x)
    ops.add_rmsnorm(x2, None, dev(w), 1e-5, out)
    assert np.array_equal(host(x2), x) and rel_err(host(out), plain.rms_norm(x, w, 1e-5)) < TOL[dtype]
    rows = np.array([7, 0, 7, 3])
    out4 = torch.empty(4, dim, device="cuda", dtype=DT[dtype])
    x3 = dev(x)
    ops.add_rmsnorm(x3, dev(delta, DT[dtype]), dev(w), 1e-5, out4, rows=dev(rows, torch.int32))
    assert np.array_equal(host(x3), x) and rel_err(host(out4), plain.rms_norm(want_x[rows], w, 1e-5)) < TOL[dtype]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rmsnorm_rows_on_a_strided_view(ops, dtype):
    rng = np.random.default_rng(1)
    x = as_stored(rng.standard_normal((20, 200)), dtype)
    w = (1 + 0.1 * rng.standard_normal(48)).astype(np.float32)
    xd = dev(x, DT[dtype])
    view = xd[:, 16:64]
    ops.rmsnorm_rows(view, dev(w), 3e-6, view)
    got = host(xd)
    assert rel_err(got[:, 16:64], plain.rms_norm(x[:, 16:64], w, 3e-6)) < TOL[dtype]
    assert np.array_equal(got[:, :16], x[:, :16]) and np.array_equal(got[:, 64:], x[:, 64:])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_silu_mul(ops, dtype):
    rng = np.random.default_rng(2)
    gu = as_stored(rng.standard_normal((11, 2 * 203)) * 4, dtype)
    out = torch.empty(11, 203, device="cuda", dtype=DT[dtype])
    ops.silu_mul(dev(gu, DT[dtype]), out)
    assert rel_err(host(out), plain.swiglu(gu[:, :203], gu[:, 203:])) < TOL[dtype]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,head_dim,theta", [(3, 48, 1e4), (5, 16, 1e6), (2, 128, 5e5)])
def test_rope(ops, dtype, heads, head_dim, theta):
    rng = np.random.default_rng(3)
    x = as_stored(rng.standard_normal((13, heads * head_dim)), dtype)
    pos = np.array([0, 1, 2, 3, 17, 100, 1000, 4095, 40000, 5, 6, 7, 8])
    xd = dev(x, DT[dtype])
    ops.rope(xd, dev(pos, torch.int32), dev(plain.rope_inv_freq(theta, head_dim)), heads, head_dim)
    assert rel_err(host(xd), plain.rope_neox(x, pos, heads, head_dim, theta)) < TOL[dtype]
    assert np.array_equal(host(xd)[0], x[0])     # position 0 is the identity


def paged_cache(rng, dtype, n_tokens_per_seq, kv_heads, head_dim, page, n_pages):
    """Keys and values of several sequences scattered over shuffled pages."""
    pages = rng.permutation(n_pages)
    kc = np.zeros((n_pages, kv_heads, page, head_dim), dtype=np.float32)
    vc = np.zeros_like(kc)
    tables, ks, vs, used = [], [], [], 0
    for n in n_tokens_per_seq:
        nb = -(-n // page)
        tab = pages[used:used + nb]
        used += nb
        k = as_stored(rng.standard_normal((n, kv_heads, head_dim)), dtype)
        v = as_stored(rng.standard_normal((n, kv_heads, head_dim)), dtype)
        for j in range(n):
            kc[tab[j // page], :, j % page] = k[j]
            vc[tab[j // page], :, j % page] = v[j]
        tables.append(tab), ks.append(k), vs.append(v)
    mb = max(len(t) for t in tables) + 3
    bt = np.zeros((len(tables), mb), dtype=np.int32)
    for i, t in enumerate(tables):
        bt[i, :len(t)] = t
    return kc, vc, bt, ks, vs


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("T", [21, 300])
@pytest.mark.parametrize("Hq,Hkv,Dh", [(6, 3, 48), (4, 2, 64), (5, 3, 64), (8, 2, 128), (3, 1, 128), (2, 1, 256)])
def test_kv_append_and_fused_norm_rope_append(ops, dtype, T, Hq, Hkv, Dh):
    """Head size 48 runs the general kernel, 64 / 128 / 256 the one that holds a head in a warp's registers, and
    with hundreds of tokens the one that works on a token's heads side by side (odd head counts put a query head
    and a key head, or a value head and nothing, into one warp)."""
    rng = np.random.default_rng(4)
    page = 8
    n_pages = max(12, T // page + 5)
    qkv = as_stored(rng.standard_normal((T, (Hq + 2 * Hkv) * Dh)), dtype)
    qw, kw = (1 + 0.2 * rng.standard_normal(Dh)).astype(np.float32), (1 + 0.2 * rng.standard_normal(Dh)).astype(np.float32)
    pos = rng.integers(0, 3000, T)
    slots = rng.permutation(n_pages * page)[:T]
    slots[5] = -1                                  # a padding row writes nothing
    kc = torch.zeros(n_pages, Hkv, page, Dh, device="cuda", dtype=DT[dtype])
    vc = torch.zeros_like(kc)
    inv = plain.rope_inv_freq(1e6, Dh)
    qd = dev(qkv, DT[dtype])
    ops.qk_norm_rope_append(qd, dev(qw), dev(kw), 1e-6, 1e-5, dev(inv), dev(pos, torch.int32), dev(slots, torch.int32),
                            kc, vc, Hq, Hkv, Dh)
    q, k, v = qkv[:, :Hq * Dh], qkv[:, Hq * Dh:(Hq + Hkv) * Dh], qkv[:, (Hq + Hkv) * Dh:]
    want_q = plain.rope_neox(plain.rms_norm(q.reshape(T * Hq, Dh), qw, 1e-6).reshape(T, -1), pos, Hq, Dh, 1e6)
    want_k = plain.rope_neox(plain.rms_norm(k.reshape(T * Hkv, Dh), kw, 1e-5).reshape(T, -1), pos, Hkv, Dh, 1e6)
    assert rel_err(host(qd)[:, :Hq * Dh], want_q) < TOL[dtype]
    got_k, got_v = host(kc), host(vc)
    for t in range(T):
        if slots[t] < 0:
            continue
        p, o = slots[t] // page, slots[t] % page
        assert rel_err(got_k[p, :, o].reshape(1, -1), want_k[t].reshape(1, -1)) < TOL[dtype]
        assert np.array_equal(got_v[p, :, o].reshape(-1), v[t])
    written = {(s // page, s % page) for s in slots if s >= 0}
    for p in range(n_pages):
        for o in range(page):
            if (p, o) not in written:
                assert not got_k[p, :, o].any() and not got_v[p, :, o].any()
    # the unfused kernel writes the same places
    kc2, vc2 = torch.zeros_like(kc), torch.zeros_like(vc)
    ops.kv_append(dev(want_k, DT[dtype]), dev(v, DT[dtype]), dev(slots, torch.int32), kc2, vc2)
    assert np.array_equal(host(vc2), got_v)
    # without norm weights and without rotation the fused kernel only copies
    q2 = dev(qkv, DT[dtype])
    ops.qk_norm_rope_append(q2, None, None, 0, 0, None, dev(pos, torch.int32), dev(slots, torch.int32), kc2, vc2, Hq, Hkv, Dh)
    assert np.array_equal(host(q2), qkv)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("M,N,K", [(1, 503, 96), (3, 72, 200), (8, 1000, 520), (13, 311, 144), (70, 130, 75), (200, 96, 1000)])
def test_gemm_simt(ops, dtype, M, N, K):
    rng = np.random.default_rng(M * N)
    a, w = as_stored(rng.standard_normal((M, K)), dtype), as_stored(rng.standard_normal((N, K)), dtype)
    out = torch.empty(M, N, device="cuda", dtype=DT[dtype])
    ops.gemm_simt(dev(a, DT[dtype]), dev(w, DT[dtype]), out)
    assert rel_err(host(out), plain.linear(a, w)) < TOL[dtype]
    if dtype == "bfloat16":                         # logits come out in float32
        out32 = torch.empty(M, N, device="cuda")
        ops.gemm_simt(dev(a, DT[dtype]), dev(w, DT[dtype]), out32)
        assert rel_err(host(out32), plain.linear(a, w)) < 2e-5


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("M,N,K", [(1, 1, 2048), (4, 7, 1016), (5, 33, 2056), (8, 300, 1024), (16, 32, 2048), (9, 600, 512), (16, 1184, 4096)])
def test_few_rows_with_k_shared_by_warps(ops, dtype, M, N, K):
    """One, two, four and eight warps a column: columns that leave warps over, k's that give the last warps less or nothing.
    A row's sums do not depend on how many rows there are."""
    rng = np.random.default_rng(M + N + K)
    a, w = as_stored(rng.standard_normal((M, K)), dtype), as_stored(rng.standard_normal((N, K)), dtype)
    da, dw = dev(a, DT[dtype]), dev(w, DT[dtype])
    out, row = torch.full((M, N), float("nan"), device="cuda"), torch.empty(1, N, device="cuda")
    ops.gemm_simt(da, dw, out)
    assert rel_err(host(out), plain.linear(a, w)) < 2e-5
    ops.gemm_simt(da[-1:], dw, row)
    assert torch.equal(row[0], out[-1])


@pytest.mark.parametrize("tile,splits", [(t, c) for t in range(3) for c in (1, 2, 4, 8)])
@pytest.mark.parametrize("M,N,K", [(17, 1, 1), (33, 65, 37), (129, 63, 260), (64, 64, 1024), (97, 200, 1504)])
def test_float_products_in_every_tiling(ops, tile, splits, M, N, K):
    """Tiles' edges, widths whose rows are no whole 16-byte pieces, splits that get no slice of k; a row stride above the row."""
    from tiny_inference_engine_b200.ops.library import call
    rng = np.random.default_rng(M + N + K)
    a, w = rng.standard_normal((M, K + 4)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32)
    da, dw, out = dev(a), dev(w), torch.full((M, N + 3), -7.0, device="cuda")
    call("tie_gemm_f32_tiled", da.data_ptr(), dw.data_ptr(), out.data_ptr(), M, N, K, K + 4, K, N + 3, tile, splits,
         torch.cuda.current_stream().cuda_stream)
    assert rel_err(host(out)[:, :N], plain.linear(a[:, :K], w)) < TOL["float32"]
    assert (host(out)[:, N:] == -7.0).all()


@pytest.mark.parametrize("bn,splits", [(32, 1), (32, 8), (64, 1), (64, 4), (96, 1), (96, 2), (96, 8)])
@pytest.mark.parametrize("M,N,K,pad", [(1, 1, 64, 0), (129, 97, 130, 4), (128, 96, 1024, 0), (300, 200, 1031, 1)])
def test_float_products_by_three_terms(ops, bn, splits, M, N, K, pad):
    """Edges of tiles, k-blocks that end early, splits that get no k-block, rows that are no whole 16-byte pieces. The bound is twice the
    largest error measured (1.1e-7 at k = 4,096; csrc/gemm_f32_split.cu has the figures, the FFMAs' too)."""
    from tiny_inference_engine_b200.ops.library import call
    rng = np.random.default_rng(M + N + K)
    a, w = rng.standard_normal((M, K + pad)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32)
    da, dw, out = dev(a), dev(w), torch.full((M, N + 3), -7.0, device="cuda")
    call("tie_gemm_f32_split", da.data_ptr(), dw.data_ptr(), out.data_ptr(), M, N, K, K + pad, K, N + 3, bn, splits,
         torch.cuda.current_stream().cuda_stream)
    want = a[:, :K].astype(np.float64) @ w.astype(np.float64).T
    got = host(out)
    assert np.linalg.norm(got[:, :N] - want) < 2.2e-7 * np.linalg.norm(want) and (got[:, N:] == -7.0).all()


@pytest.mark.parametrize("bn,splits", [(64, 1), (96, 4)])
def test_float_products_by_three_terms_of_infinities_and_large_values(ops, bn, splits):
    """An infinity, a NaN or a value that bfloat16 would round to an infinity reaches exactly the outputs it belongs to."""
    from tiny_inference_engine_b200.ops.library import call
    rng = np.random.default_rng(bn)
    M, N, K = 200, 150, 520
    a, w = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32)
    w[w == 0] = 1.0
    w[3, 40] = 1.0
    a[5, 40], a[130, 300], a[7, 519], w[60, 65], a[9, :], a[9, 2] = np.inf, -np.inf, np.nan, np.inf, 0.0, 3.4e38
    w[:, 2] = np.clip(w[:, 2], -0.5, 0.5)
    da, dw, out = dev(a), dev(w), torch.empty(M, N, device="cuda")
    call("tie_gemm_f32_split", da.data_ptr(), dw.data_ptr(), out.data_ptr(), M, N, K, K, K, N, bn, splits, torch.cuda.current_stream().cuda_stream)
    got, want = host(out).astype(np.float64), torch.from_numpy(a).double() @ torch.from_numpy(w).double().T
    want = want.numpy()
    odd = ~np.isfinite(want)
    assert odd.sum() > 400 and ((got[odd] == want[odd]) | (np.isnan(got[odd]) & np.isnan(want[odd]))).all()
    rest = (~odd) & (np.arange(M) != 9)[:, None]
    assert np.linalg.norm(got[rest] - want[rest]) < 1e-6 * np.linalg.norm(want[rest])
    assert (np.abs(got[9] - want[9])[~odd[9]] <= 1e-6 * np.abs(want[9])[~odd[9]]).all()


def float_products_both_ways(a, w, bn, splits):
    """out = a w^T by three terms and by FFMAs (64 x 64 tiles, whole k), and the relative errors of both against 64 bits."""
    from tiny_inference_engine_b200.ops.library import call
    M, K, N = *a.shape, w.shape[0]
    outs = [torch.empty(M, N, device="cuda") for _ in range(2)]
    for name, out, tile, s in (("tie_gemm_f32_split", outs[0], bn, splits), ("tie_gemm_f32_tiled", outs[1], 1, 1)):
        call(name, a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, K, K, N, tile, s, torch.cuda.current_stream().cuda_stream)
    want = a.double() @ w.double().T
    return outs[0], want, *(float((o.double() - want).norm() / want.norm()) for o in outs)


@pytest.mark.parametrize("size", [1.0, 1e-35, 3e-37, 1e-40])
@pytest.mark.parametrize("bn,splits", [(32, 1), (96, 2)])
def test_float_products_by_three_terms_of_small_values(ops, bn, splits, size):
    """Operands whose low bits bfloat16 has no exponent for (below 2^-109), and subnormal ones: no bit of them is lost, the error is
    no larger than with FFMAs (results near the smallest float round alike in both)."""
    g = torch.Generator("cuda").manual_seed(3)
    a, w = (torch.randn(n, 600, device="cuda", generator=g) for n in (130, 100))
    _, _, terms, ffma = float_products_both_ways(a * size, w, bn, splits)
    assert terms <= ffma


@pytest.mark.parametrize("K", [128, 200, 1024, 4096])
@pytest.mark.parametrize("kind", ["normal", "one sign", "even", "near one"])
def test_float_products_are_nearer_to_64_bits_than_ffmas(ops, kind, K):
    """What `gemm` picks for 192 rows against the FFMA kernel with whichever of its tilings is nearest, on operands of either and of one
    sign: the tensor core's additions cut off, which for sums of one sign was an error of its own (0.9 to 1.0e-7)."""
    from tiny_inference_engine_b200.ops.library import call
    g = torch.Generator("cuda").manual_seed(K)
    M, N = 192, 256
    a, w = (torch.randn(n, K, device="cuda", generator=g) for n in (M, N))
    if kind != "normal":
        a, w = {"one sign": (a.abs(), w.abs()), "even": (a.sigmoid(), w.sigmoid()), "near one": (1.0 + 0.01 * a, 1.0 + 0.01 * w)}[kind]
    want = a.double() @ w.double().T
    off = lambda o: float((o.double() - want).norm() / want.norm())      # noqa: E731
    out = torch.empty(M, N, device="cuda")
    ops.gemm(a, w, out)
    best = 1.0
    for tile in (0, 1, 2):
        for splits in (1, 2, 4, 8):
            if K // 32 // splits >= 4:
                ffma = torch.empty(M, N, device="cuda")
                call("tie_gemm_f32_tiled", a.data_ptr(), w.data_ptr(), ffma.data_ptr(), M, N, K, K, K, N, tile, splits, torch.cuda.current_stream().cuda_stream)
                best = min(best, off(ffma))
    assert off(out) <= best


@pytest.mark.parametrize("M,N,K", [(17, 512, 1024), (32, 1024, 2048), (24, 16384, 128), (33, 16384, 128), (17, 14208, 320), (17, 24000, 400)])
def test_float_products_of_few_rows(ops, M, N, K):
    """Products on either side of the line between the two float kernels, and those whose clusters were taken for more than are resident."""
    g = torch.Generator("cuda").manual_seed(N)
    a, w = (torch.randn(n, K, device="cuda", generator=g) for n in (M, N))
    out = torch.full((M, N), float("nan"), device="cuda")
    ops.gemm(a, w, out)
    want = a.double() @ w.double().T
    assert float((out.double() - want).norm() / want.norm()) < 4e-7


def test_float_products_by_three_terms_whose_partial_sums_overflow(ops):
    """All terms as large as they get: 2^16 times the products of the low ones adds up to three times the result, beyond the largest
    float, where the result is below it."""
    x = (1.0 + 254 / 256 * 2.0 ** -8 + 126 / 128 * 2.0 ** -16) * 2.0 ** 60
    a = torch.zeros(70, 200, device="cuda")
    a[:, :64] = x
    w = torch.full((40, 200), 2.0 * x, device="cuda")
    out, want, terms, _ = float_products_both_ways(a, w, 32, 1)
    assert torch.isfinite(out).all() and terms < 1e-6


def test_a_float_product_may_be_captured_before_any_other_has_run(ops):
    """In a process of its own: the first product of all inside a graph's capture, as the FFMA kernels allow."""
    import pathlib
    import subprocess
    import sys
    script = """
import torch
from tiny_inference_engine_b200 import ops
from tiny_inference_engine_b200.ops.library import library
library()
a, w, out = (torch.randn(n, k, device="cuda") for n, k in ((64, 512), (96, 512), (64, 96)))
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    ops.gemm(a, w, out)
graph.replay()
torch.cuda.synchronize()
want = a.double() @ w.double().T
assert float((out.double() - want).norm() / want.norm()) < 4e-7
"""
    done = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300,
                          cwd=pathlib.Path(__file__).resolve().parents[1])
    assert done.returncode == 0, done.stderr[-2000:]


def dense_reference(q, k, v, Hq, Hkv, Dh, n_new, window=0):
    """The last n_new rows of causal attention over all of k, v."""
    n = k.shape[0]
    qfull = np.zeros((n, Hq * Dh))
    qfull[n - n_new:] = q
    return plain.causal_attention(qfull, k.reshape(n, -1), v.reshape(n, -1), Hq, Hkv, Dh, window)[n - n_new:]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("Hq,Hkv,Dh,page,window", [(4, 2, 16, 16, 0), (8, 1, 32, 8, 0), (3, 3, 48, 32, 0), (6, 2, 128, 16, 0),
                                                  (5, 5, 80, 4, 0), (4, 1, 64, 16, 37)])
def test_paged_attention_rows_and_split(ops, dtype, Hq, Hkv, Dh, page, window):
    """Mixed batch: two sequences bring portions over a cached prefix, three bring one token;
    pages are scattered. Rows kernel for the first, split kernel for the others."""
    rng = np.random.default_rng(Hq * Dh)
    ctx = [45, 300, 1, 33, 700]          # tokens in the cache after the step
    new = [45, 17, 1, 1, 1]              # of which this step brings
    kc, vc, bt, ks, vs = paged_cache(rng, dtype, ctx, Hkv, Dh, page, 120 * 16 // page)
    T = sum(new)
    q = as_stored(rng.standard_normal((T, Hq * Dh)), dtype)
    qs = np.concatenate([[0], np.cumsum(new)])
    scale = 1.0 / np.sqrt(Dh)
    want = np.concatenate([dense_reference(q[qs[i]:qs[i + 1]], ks[i], vs[i], Hq, Hkv, Dh, new[i], window) for i in range(5)])
    seq_of_row = np.repeat(np.arange(5), new)
    out = torch.zeros(T, Hq * Dh, device="cuda", dtype=DT[dtype])
    args = (dev(kc, DT[dtype]), dev(vc, DT[dtype]), out)
    meta = (dev(qs, torch.int32), dev(np.array(ctx), torch.int32), dev(bt, torch.int32))
    ops.attention_rows(dev(q, DT[dtype]), *args, dev(seq_of_row, torch.int32), *meta, Hq, Hkv, Dh, scale, window)
    assert rel_err(host(out), want) < TOL[dtype]
    # the same single-token sequences through the split kernel, with splits of 64 keys
    out2 = torch.zeros_like(out)
    n_multi = new[0] + new[1]
    scratch = torch.empty(ops.attention_split_scratch_floats(3, Hq, Dh, 11), device="cuda")
    ops.attention_split(dev(q, DT[dtype]), *args[:2], out2, *meta, Hq, Hkv, Dh, scale, dev(np.array([2, 3, 4]), torch.int32),
                        3, 64, 11, scratch, window)
    assert rel_err(host(out2)[n_multi:], want[n_multi:]) < TOL[dtype]
    assert not host(out2)[:n_multi].any()


@pytest.mark.parametrize("Hq,Hkv,Dh,page,window,new,ctx", [
    (4, 2, 128, 16, 0, [16, 3, 40], [16, 70, 40]), (2, 1, 64, 8, 0, [1, 15, 33], [97, 15, 64]), (3, 3, 32, 12, 9, [31, 17], [31, 90]),
    (2, 2, 128, 4, 33, [50], [140])])
def test_float_rows_by_tiles(ops, Hq, Hkv, Dh, page, window, new, ctx):
    """Tiles of 16 rows and 32 keys with several sequences in one, portions behind cached keys, windows; and a token with NaN values
    leaves the rows before it, and the other sequences, as they are."""
    rng = np.random.default_rng(Hq * Dh + window)
    kc, vc, bt, ks, vs = paged_cache(rng, "float32", ctx, Hkv, Dh, page, 60 * 16 // page)
    T, qs = sum(new), np.concatenate([[0], np.cumsum(new)])
    q = rng.standard_normal((T, Hq * Dh)).astype(np.float32) * 3
    want = np.concatenate([dense_reference(q[qs[i]:qs[i + 1]], ks[i], vs[i], Hq, Hkv, Dh, new[i], window) for i in range(len(new))])
    args = (dev(np.repeat(np.arange(len(new)), new), torch.int32), dev(qs, torch.int32), dev(np.array(ctx), torch.int32), dev(bt, torch.int32))
    out = torch.full((T, Hq * Dh), float("nan"), device="cuda")
    ops.attention_rows(dev(q), dev(kc), dev(vc), out, *args, Hq, Hkv, Dh, 1.0 / np.sqrt(Dh), window)
    assert rel_err(host(out), want) < TOL["float32"]
    sick = ctx[-1] - 2                                 # the second last token of the last sequence
    vc = vc.copy()
    vc[bt[len(new) - 1, sick // page], :, sick % page] = np.nan
    ops.attention_rows(dev(q), dev(kc), dev(vc), out, *args, Hq, Hkv, Dh, 1.0 / np.sqrt(Dh), window)
    assert rel_err(host(out)[:T - 2], want[:T - 2]) < TOL["float32"]
    assert np.isnan(host(out)[T - 2:]).all()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("far", [0, 15, 16, 31, 32, 255, 256, 257, 511, 512, 1022, 1023])
def test_one_far_key_among_a_thousand_is_found(ops, dtype, far):
    """The query matches exactly one key, at a page's edge, a chunk's edge, a split's edge, the
    first key, the last: the output must be that key's value row. Random data would hide a key
    that is skipped or read from the wrong page: it would move the result by a thousandth."""
    rng = np.random.default_rng(far)
    Hq, Hkv, Dh, page, n = 4, 2, 32, 16, 1024
    kc, vc, bt, ks, vs = paged_cache(rng, dtype, [n], Hkv, Dh, page, 80)
    q = np.zeros((1, Hq * Dh), dtype=np.float32)
    for h in range(Hq):
        q[0, h * Dh:(h + 1) * Dh] = 8.0 * ks[0][far, h // 2] * np.sqrt(Dh)   # score ~ 8 * |k|^2 ~ 256 above the rest
    q = as_stored(q, dtype)
    meta = (dev(np.array([0, 1]), torch.int32), dev(np.array([n]), torch.int32), dev(bt, torch.int32))
    one_hot = np.concatenate([vs[0][far, h // 2] for h in range(Hq)])[None]
    want = dense_reference(q, ks[0], vs[0], Hq, Hkv, Dh, 1)
    assert np.abs(want - one_hot).max() < 1e-3      # the far key really holds all the weight
    for split in (False, True):
        out = torch.zeros(1, Hq * Dh, device="cuda", dtype=DT[dtype])
        if split:
            scratch = torch.empty(ops.attention_split_scratch_floats(1, Hq, Dh, 4), device="cuda")
            ops.attention_split(dev(q, DT[dtype]), dev(kc, DT[dtype]), dev(vc, DT[dtype]), out, *meta, Hq, Hkv, Dh,
                                1 / np.sqrt(Dh), dev(np.array([0]), torch.int32), 1, 256, 4, scratch)
        else:
            ops.attention_rows(dev(q, DT[dtype]), dev(kc, DT[dtype]), dev(vc, DT[dtype]), out,
                               dev(np.array([0]), torch.int32), *meta, Hq, Hkv, Dh, 1 / np.sqrt(Dh))
        assert np.abs(host(out) - want).max() < 1e-2, f"split={split}"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_window_edge(ops, dtype):
    """With a window of 40 the key at position pos-39 counts and the one at pos-40 does not."""
    rng = np.random.default_rng(9)
    Hq, Hkv, Dh, page, n, window = 2, 1, 32, 8, 200, 40
    kc, vc, bt, ks, vs = paged_cache(rng, dtype, [n], Hkv, Dh, page, 40)
    meta = (dev(np.array([0, 1]), torch.int32), dev(np.array([n]), torch.int32), dev(bt, torch.int32))
    for target, inside in ((n - 1 - 39, True), (n - 1 - 40, False)):
        q = as_stored(np.tile(8.0 * ks[0][target, 0] * np.sqrt(Dh), Hq)[None], dtype)
        out = torch.zeros(1, Hq * Dh, device="cuda", dtype=DT[dtype])
        ops.attention_rows(dev(q, DT[dtype]), dev(kc, DT[dtype]), dev(vc, DT[dtype]), out, dev(np.array([0]), torch.int32),
                           *meta, Hq, Hkv, Dh, 1 / np.sqrt(Dh), window)
        hit = np.abs(host(out)[0, :Dh] - vs[0][target, 0]).max() < 1e-2
        assert hit == inside


def test_sampling_kernel_greedy_and_temperature(ops):
    rng = np.random.default_rng(5)
    R, V = 7, 1531
    z = (rng.standard_normal((R, V)) * 2).astype(np.float32)
    z[2, 100] = z[2, 900] = z[2].max() + 1          # a tie goes to the lowest id
    z[3, 5] = np.inf
    out = torch.empty(R, dtype=torch.int32, device="cuda")
    ops.sample(dev(z), out)
    assert out.tolist() == [plain.sample(z[r]) for r in range(R)] and out[2].item() == 100
    temps = np.array([0.8, 0.0, 1.0, 0.7, 1e-45, 2.5, 0.3], dtype=np.float32)
    with np.errstate(divide="ignore", over="ignore"):
        inv = np.where(temps > 0, np.float32(1) / temps, 0).astype(np.float32)
    inv[~np.isfinite(inv)] = 0
    seeds = np.array([7, 1, 2 ** 63 + 11, 4, 5, 6, 2 ** 40], dtype=np.uint64)
    for counter in (0, 1, 2, 1000, 2 ** 33):
        ctr = np.full(R, counter, dtype=np.int64)
        ops.sample(dev(z), out, dev(inv), torch.from_numpy(seeds.view(np.int64)).cuda(), dev(ctr, torch.int64))
        want = [plain.sample(z[r], float(temps[r]), u=plain.uniform_for(int(seeds[r]), counter)) for r in range(R)]
        assert out.tolist() == want


def test_sampling_kernel_frequencies(ops):
    z = np.tile(np.array([[0.0, 1.0, 2.0, -30.0, 0.5]], dtype=np.float32), (2000, 1))
    out = torch.empty(2000, dtype=torch.int32, device="cuda")
    inv = np.full(2000, 1 / 0.8, dtype=np.float32)
    ops.sample(dev(z), out, dev(inv), dev(np.full(2000, 3), torch.int64), dev(np.arange(2000), torch.int64))
    p = np.exp(z[0] / 0.8 - (z[0] / 0.8).max())
    p /= p.sum()
    assert np.abs(np.bincount(out.cpu().numpy(), minlength=5) / 2000 - p).max() < 0.03


def _filtered_case(ops, z, rows, counter, one_cta=False):
    """rows: (temperature, top_k, top_p, seed) for each row of z; the kernels against the sampler on the host."""
    from tiny_inference_engine_b200.sampling import SamplingParams
    from host_sampler import sample_host
    R = len(rows)
    params = [SamplingParams(temperature=t, top_k=k, top_p=p, seed=s) for t, k, p, s in rows]
    inv = np.array([q.inv_temperature() for q in params], dtype=np.float32)
    seeds = np.array([q.seed for q in params], dtype=np.uint64)
    out = torch.full((R,), -1, dtype=torch.int32, device="cuda")
    ops.sample(dev(z), out, dev(inv), torch.from_numpy(seeds.view(np.int64)).cuda(), dev(np.full(R, counter), torch.int64),
               dev(np.array([q.top_k for q in params]), torch.int32), dev(np.array([q.top_p for q in params], dtype=np.float32)),
               one_cta=one_cta)
    want = [sample_host(z[r], params[r], counter) for r in range(R)]
    assert out.tolist() == want, [(rows[r], out[r].item(), want[r]) for r in range(R) if out[r].item() != want[r]]


@pytest.mark.parametrize("one_cta", [False, True])
def test_sampling_kernel_top_k_and_top_p(ops, one_cta):
    """Few kept candidates are sorted in shared memory; more than 1,024, or top-p alone, are found by selection
    over the whole row. Equal logits are taken in id order; -inf logits weigh nothing. Both kernels: the cluster of
    8 CTAs a row, and the one-CTA kernel of the largest vocabularies."""
    rng = np.random.default_rng(11)
    V = 1531
    rows = []
    for k in (0, 1, 5, 200, 1024, 1100, V, 5000):
        for p in (1.0, 0.9, 0.3, 1e-6):
            rows.append((float(rng.choice([0.3, 0.8, 1.0, 2.5])), k, p, int(rng.integers(0, 2 ** 62))))
    rows += [(0.0, 5, 0.5, 3), (1e-45, 5, 0.5, 3)]                       # greedy whatever the filters say
    R = len(rows)
    z = (rng.standard_normal((R, V)) * 2.5).astype(np.float32)
    z[:, 40:60] = z[:, 700:701]                                          # twenty equal logits in every row
    z[::3, 100:400] = -np.inf
    z[5] = 0.25                                                          # a row of equal logits: the cut falls among ties
    z[6] = np.round(z[6])                                                # many ties at every value
    for counter in (0, 1, 2, 3, 77, 2 ** 33):
        _filtered_case(ops, z, rows, counter, one_cta)
    z[7, 3] = np.inf                                                     # a certain token
    _filtered_case(ops, z, rows, 5, one_cta)


def test_sampling_kernel_filters_over_a_large_vocabulary(ops):
    rng = np.random.default_rng(12)
    V = 151936
    rows = [(0.7, 20, 0.8, 1), (0.7, 0, 0.9, 2), (1.0, 5000, 0.95, 3), (1.3, 0, 0.5, 4), (0.7, 20, 1.0, 5), (1.0, 2000, 1.0, 6)]
    z = (rng.standard_normal((len(rows), V)) * np.array([3, 3, 0.01, 0.01, 5, 1])[:, None]).astype(np.float32)
    for counter in (0, 1, 2):
        _filtered_case(ops, z, rows, counter)
    _filtered_case(ops, z, rows, 3, one_cta=True)


@pytest.mark.parametrize("one_cta", [False, True])
def test_sampling_kernels_refuse_rows_with_a_nan_or_nothing_finite(ops, one_cta):
    """The reference's sampler raises for a NaN logit and for a row of -inf (src/sampling/sampler.cpp:18-26). The
    kernels answer -2 for such a row, with or without filters, and sample the rows beside it as ever."""
    from host_sampler import sample_host
    from tiny_inference_engine_b200.errors import InvalidArgument
    from tiny_inference_engine_b200.sampling import SamplingParams
    rng = np.random.default_rng(21)
    V = 3001
    params = [SamplingParams(temperature=t, top_k=k, top_p=p, seed=7 + i) for i, (t, k, p) in enumerate(
        [(0.0, 0, 1.0), (0.0, 0, 1.0), (0.8, 0, 1.0), (0.8, 0, 1.0), (0.8, 20, 0.9), (0.8, 20, 0.9), (0.8, 20, 0.9),
         (1.0, 0, 0.5), (1.0, 0, 0.5), (0.0, 0, 1.0), (0.7, 5, 1.0)])]
    R = len(params)
    z = (rng.standard_normal((R, V)) * 2).astype(np.float32)
    z[1, 2999] = np.nan          # greedy, a NaN at the far end of the row
    z[3, 0] = np.nan             # temperature, a NaN at the start
    z[5, 1500] = np.nan          # filtered, a NaN in the middle (and a +inf, which does not save the row)
    z[5, 7] = np.inf
    z[6] = -np.inf               # filtered, nothing finite
    z[8] = np.nan                # every logit a NaN
    z[9] = -np.inf               # greedy, nothing finite
    z[10, 5:] = -np.inf          # five finite values left: this row is fine
    refused = {1, 3, 5, 6, 8, 9}
    for r in range(R):
        if r in refused:
            with pytest.raises(InvalidArgument):
                sample_host(z[r], params[r], 3)
    out = torch.full((R,), 77, dtype=torch.int32, device="cuda")
    seeds = np.array([q.seed for q in params], dtype=np.int64)
    ops.sample(dev(z), out, dev(np.array([q.inv_temperature() for q in params], dtype=np.float32)), dev(seeds, torch.int64),
               dev(np.full(R, 3), torch.int64), dev(np.array([q.top_k for q in params]), torch.int32),
               dev(np.array([q.top_p for q in params], dtype=np.float32)), one_cta=one_cta)
    got = out.tolist()
    assert got == [-2 if r in refused else sample_host(z[r], params[r], 3) for r in range(R)]


def test_the_constants_the_host_plans_with_are_the_kernels_own(ops):
    from tiny_inference_engine_b200.ops.library import library
    from tiny_inference_engine_b200.parts import attention as att
    lib = library()
    assert att.TMA_DECODE_TABLE_ENTRIES == lib.tie_attention_decode_limit(0)
    assert att.MAX_SPLITS <= lib.tie_attention_decode_limit(1)
    assert att.NUM_SMS == torch.cuda.get_device_properties(0).multi_processor_count
    assert 1 <= lib.tie_gemm_tc2_pairs() <= att.NUM_SMS // 2


def test_refusals_are_clear(ops):
    from tiny_inference_engine_b200.errors import InvalidArgument
    q = torch.zeros(1, 2 * 20, device="cuda")
    kc = torch.zeros(4, 1, 8, 20, device="cuda")
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    with pytest.raises(InvalidArgument, match="head_dim 20 must be a multiple of 8"):
        ops.attention_rows(q, kc, kc.clone(), torch.zeros_like(q), i32(0), i32(0, 1), i32(1), i32(0, 0).view(1, 2), 2, 1, 20, 1.0)
    with pytest.raises(InvalidArgument, match="not a multiple"):
        ops.attention_rows(torch.zeros(1, 48, device="cuda"), torch.zeros(4, 2, 8, 16, device="cuda"),
                           torch.zeros(4, 2, 8, 16, device="cuda"), torch.zeros(1, 48, device="cuda"), i32(0), i32(0, 1),
                           i32(1), i32(0, 0).view(1, 2), 3, 2, 16, 1.0)
    with pytest.raises(InvalidArgument, match="CUDA tensors"):
        ops.silu_mul(torch.zeros(2, 8), torch.zeros(2, 4))
    with pytest.raises(InvalidArgument, match="shapes"):
        ops.gemm_simt(torch.zeros(2, 8, device="cuda"), torch.zeros(4, 9, device="cuda"), torch.zeros(2, 4, device="cuda"))


@pytest.mark.parametrize("out_dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("M,N,K", [(1, 503, 96), (3, 311, 144), (8, 1000, 520), (16, 72, 200), (33, 300, 64), (77, 130, 1000),
                                   (128, 256, 512), (200, 96, 72), (300, 503, 96), (700, 311, 136), (513, 256, 64),
                                   (1100, 777, 520)])
def test_gemm_tensor_cores(ops, out_dtype, M, N, K):
    """tcgen05 product with the tiling the engine would pick, at sizes that end inside a tile in
    every direction (rows, columns, k)."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(M + N + K)
    a, w = as_stored(rng.standard_normal((M, K)), "bfloat16"), as_stored(rng.standard_normal((N, K)), "bfloat16")
    out = torch.full((M, N), float("nan"), device="cuda", dtype=DT[out_dtype])
    ops.gemm(dev(a, torch.bfloat16), dev(w, torch.bfloat16), out)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(out), plain.linear(a, w)) < (TOL["bfloat16"] if out_dtype == "bfloat16" else 2e-5)


@pytest.mark.parametrize("M,N,K", [(1, 503, 96), (8, 1000, 520), (16, 72, 200), (77, 130, 1000), (128, 256, 512), (200, 96, 72),
                                   (300, 503, 96), (700, 311, 136), (1100, 2560, 520)])
def test_products_with_the_weight_kept_in_k_blocks(ops, M, N, K):
    """A bound product keeps its weight as [ceil(K / 64), N, 64] (every box a stage loads is one piece of memory) and
    gives the plain product at every token count: the transposed tiling, the 128-token row tiles, the kernel on pairs
    of SMs (the last case), widths and depths that end inside a tile (rows of the next k-block come in with the
    last boxes; they reach no output), a depth that is no multiple of 64 (zeros); and a slice of its rows
    (the k rows of a stacked q/k/v weight) without a copy."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(M * N + K)
    a, w = as_stored(rng.standard_normal((M, K)), "bfloat16"), as_stored(rng.standard_normal((N, K)), "bfloat16")
    g = ops.bound_gemm(dev(w, torch.bfloat16))
    assert g.packed_rows == N and tuple(g.w.shape) == (-(-K // 64), N, 64) and (g.N, g.K) == (N, K)
    assert torch.equal(g.row_major().cpu(), dev(w, torch.bfloat16).cpu())
    want = plain.linear(a, w)
    for out_dtype in ("bfloat16", "float32"):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=DT[out_dtype])
        got = g(dev(a, torch.bfloat16), out)
        torch.cuda.synchronize()
        gemm_select.check_status()
        assert got is out and rel_err(host(out), want) < (TOL["bfloat16"] if out_dtype == "bfloat16" else 2e-5), out_dtype
    lo, hi = N // 3, N // 3 + max(8, N // 2)
    part = g.rows(lo, hi)
    assert part.w.data_ptr() == g.w.data_ptr() and (part.N, part.row0) == (hi - lo, lo)
    wide = torch.full((M, hi - lo + 16), 7.0, device="cuda", dtype=torch.float32)
    part(dev(a, torch.bfloat16), wide[:, 8:8 + hi - lo])
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(wide[:, 8:8 + hi - lo]), want[:, lo:hi]) < 2e-5
    assert (wide[:, :8] == 7).all() and (wide[:, 8 + hi - lo:] == 7).all()


@pytest.mark.parametrize("bn", [128, 160, 192, 224, 256])
def test_pair_kernel_at_every_tile_width(ops, bn):
    """The product on pairs of SMs with tiles of 256 rows by 128 to 256 columns, plain and with the SiLU epilogue,
    at sizes that end inside a tile; the width changes which CTA computes what, not what is computed."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(bn)
    M, N, K = 600, 1000, 264
    a, w = as_stored(rng.standard_normal((M, K)), "bfloat16"), as_stored(rng.standard_normal((N, K)), "bfloat16")
    wide = torch.full((M, N + 16), 7.0, device="cuda", dtype=torch.float32)
    gemm_select.gemm_tc(dev(a, torch.bfloat16), dev(w, torch.bfloat16), wide[:, 8:8 + N], pair=True, bn=bn)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(wide[:, 8:8 + N]), plain.linear(a, w)) < 2e-5
    assert (wide[:, :8] == 7).all() and (wide[:, 8 + N:] == 7).all()
    I = 352
    gate, up = as_stored(rng.standard_normal((I, K)) * 0.3, "bfloat16"), as_stored(rng.standard_normal((I, K)) * 0.3, "bfloat16")
    out = torch.full((M, I), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm_select.gemm_tc(dev(a, torch.bfloat16), ops.interleave_gate_up(dev(gate, torch.bfloat16), dev(up, torch.bfloat16)), out,
                        silu=True, pair=True, bn=bn)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(out), plain.swiglu(plain.linear(a, gate), plain.linear(a, up))) < TOL["bfloat16"]


@pytest.mark.parametrize("M,N,K,transposed,bn,splits", [(65, 264, 72, 1, 64, 1), (129, 1001, 1096, 1, 160, 3), (256, 4992, 520, 1, 256, 1),
                                                        (200, 515, 1992, 0, 96, 4), (600, 260, 4096, 0, 64, 5), (1, 300, 136, 1, 32, 2)])
def test_pair_kernel_on_either_side_and_with_split_k(ops, M, N, K, transposed, bn, splits):
    """Pairs of SMs with the tokens or the weights on the 256-row side, k whole or split (the sums left for a consumer, or added),
    sizes that end inside a tile, rows that TMA can store and rows that it cannot (odd widths and offsets)."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(M + N + K)
    a, w = as_stored(rng.standard_normal((M, K)), "bfloat16"), as_stored(rng.standard_normal((N, K)), "bfloat16")
    want = plain.linear(a, w)
    ta, tw = dev(a, torch.bfloat16), dev(w, torch.bfloat16)
    for dtype, offset in ((torch.float32, 8), (torch.bfloat16, 8), (torch.bfloat16, 3)):
        wide = torch.full((M, N + 16), 7.0, device="cuda", dtype=dtype)
        scratch = torch.full((splits * M * N + 16,), float("nan"), device="cuda")
        gemm_select._call("tie_gemm_tc2", int(dtype == torch.bfloat16), ta.data_ptr(), tw.data_ptr(), wide[:, offset:].data_ptr(), M, N, K, K, K,
                          N + 16, 0, 0, 0, bn, transposed, splits, scratch.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        gemm_select.check_status()
        assert rel_err(host(wide[:, offset:offset + N]), want) < (TOL["bfloat16"] if dtype == torch.bfloat16 else 2e-5), (dtype, offset)
        assert (wide[:, :offset] == 7).all() and (wide[:, offset + N:] == 7).all()
        real = gemm_select._library().tie_gemm_tc_real_splits(K, splits) if splits > 1 else 0
        assert torch.isnan(scratch[real * M * N:]).all()
        if real:
            assert rel_err(scratch[:real * M * N].view(real, M, N).sum(0).cpu().numpy(), want) < 2e-5


@pytest.mark.parametrize("transposed", [0, 1])
def test_silu_epilogue_from_the_smallest_to_the_largest_gates(ops, transposed):
    """act(gate) * up against 64 bits where the exponential is 1, rounds away, and overflows; in float output, within four
    roundings of 32 bits (exp, sum, quotient, product) and the exponential's own two units."""
    from tiny_inference_engine_b200.ops import gemm_select
    gates = torch.tensor([0.0, -0.0, 1e-30, -1e-30, 0.3, -0.3, 5.0, -5.0, 17.0, -17.0, 40.0, -40.0, -43.0, -60.0, 88.0, -88.0, -88.5, -89.0,
                          -200.0, 1e38, -1e38]).to(torch.bfloat16)      # times 3 at most: below 3.4e38
    M, I, K = 100, 32, 16
    a = torch.zeros(M, K, dtype=torch.bfloat16)
    a[:, 0], a[:, 1] = gates.repeat(5)[:M], 1.5
    gate, up = torch.zeros(I, K, dtype=torch.bfloat16), torch.zeros(I, K, dtype=torch.bfloat16)
    gate[:, 0], up[:, 1] = 1.0, torch.linspace(-2, 2, I).to(torch.bfloat16)
    out = torch.full((M, I), float("nan"), device="cuda")
    w = ops.interleave_gate_up(gate.cuda(), up.cuda())
    gemm_select._call("tie_gemm_tc2", 0, a.cuda().data_ptr(), w.data_ptr(), out.data_ptr(), M, 2 * I, K, K, K, I, 1, 0, 0, 128 if transposed else 64,
                      transposed, 1, 0, 1, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    gemm_select.check_status()
    g = a[:, 0].double()
    want = (g / (1.0 + torch.exp(-g)))[:, None] * (1.5 * up[:, 1].double())[None]
    got = out.double().cpu()
    near = want.abs() > 1e-36                      # below, 32 bits have no full mantissa
    assert ((got - want).abs()[near] <= 6 * 2.0 ** -24 * want.abs()[near] * 2).all() and (got - want).abs()[~near].max() < 2e-36


@pytest.mark.parametrize("act", [1, 4, 5])
@pytest.mark.parametrize("kernel", ["pair", "pair transposed", "single", "single transposed", "split k"])
def test_silu_epilogue_of_gates_that_overflow(ops, kernel, act):
    """Gates whose sums are infinite or not a number, of every unit with a SiLU (the clamped one without a limit): in kind what
    g / (1 + exp(-g)) gives, an infinity of the same sign, NaN, or the number."""
    from tiny_inference_engine_b200.ops import gemm_select
    M, I, K = 40, 32, 128
    a = torch.zeros(M, K, dtype=torch.bfloat16)
    a[:, 0] = torch.tensor([3e38, -3e38, float("nan"), 1e38, -1e38, 104.0, 60.0, 0.0]).to(torch.bfloat16).repeat(5)
    a[:, 1] = 1.5
    gate, up = torch.zeros(I, K, dtype=torch.bfloat16), torch.zeros(I, K, dtype=torch.bfloat16)
    gate[:, 0], up[:, 1] = 2.0, torch.linspace(-1, 1, I).to(torch.bfloat16)
    w, da, out = ops.interleave_gate_up(gate.cuda(), up.cuda()), a.cuda(), torch.full((M, I), 7.0, device="cuda")
    zeros, scratch = torch.zeros(I, device="cuda"), torch.empty(2 * M * 2 * I, device="cuda")
    slope = 1.702 if act == 4 else 1.0
    unit = (zeros.data_ptr(), zeros.data_ptr(), float("inf"), slope, 0.0, 0, torch.cuda.current_stream().cuda_stream)
    sizes = (0, da.data_ptr(), w.data_ptr(), out.data_ptr(), M, 2 * I, K, K, K, I)
    if kernel.startswith("pair"):
        gemm_select._call("tie_gemm_tc2_unit", *sizes, act, 0, 0, 64, int("transposed" in kernel), 1, 0, 1, *unit)
    else:
        t = int(kernel != "single")
        splits = 2 if kernel == "split k" else 1
        gemm_select._call("tie_gemm_tc_unit", *sizes, t, 64, splits, scratch.data_ptr() if splits > 1 else 0, act, 1, 0, 0, 0, *unit)
    torch.cuda.synchronize()
    gemm_select.check_status()
    g, u = 2.0 * a[:, :1].float().expand(M, I), (1.5 * up[:, 1].float() + 0.0 * a[:, :1].float())
    if act == 4:            # its minimum and maximum, like the device's, pass over NaN
        g, u = torch.fmin(g, torch.tensor(float("inf"))), torch.fmax(u, torch.tensor(-float("inf")))
    want = g / (1.0 + torch.exp(-slope * g)) * u
    got = out.cpu()
    odd = ~torch.isfinite(want)
    assert odd.sum() == 15 * I and (torch.isnan(got) == torch.isnan(want)).all() and (got[torch.isinf(want)] == want[torch.isinf(want)]).all()
    assert ((got - want).abs()[~odd] <= 12 * 2.0 ** -24 * want.abs()[~odd] + 1e-37).all()


@pytest.mark.parametrize("act", [4, 5, 6])
@pytest.mark.parametrize("M,I,K", [(5, 48, 1024), (64, 496, 2048), (100, 48, 72), (200, 352, 264), (640, 176, 136)])
def test_gated_units_in_the_epilogue(ops, M, I, K, act):
    """The clamped unit and the ones with biases, the columns of a one and zeros behind them: k split (the unit formed where the sums are
    added), the weights or the tokens on the row side, one CTA or a pair a tile, sizes that end inside a tile."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(M + act)
    a = as_stored(rng.standard_normal((M, K)), "bfloat16")
    gate, up = (as_stored(rng.standard_normal((I, K)) * 3 / K ** 0.5, "bfloat16") for _ in range(2))
    bg, bu = rng.standard_normal(I).astype(np.float32), rng.standard_normal(I).astype(np.float32)
    ones = 0 if act == 4 else 8
    unit = gemm_select.GatedUnit(2.0, 1.702, 1.0) if act == 4 else gemm_select.GatedUnit(bias_gate=dev(bg), bias_up=dev(bu), ones=ones)
    product = ops.bound_gemm(ops.interleave_gate_up(dev(gate, torch.bfloat16), dev(up, torch.bfloat16)), silu=act, unit=unit)
    wide = torch.full((M, I + ones + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    product(dev(a, torch.bfloat16), wide[:, :I])
    torch.cuda.synchronize()
    gemm_select.check_status()
    g, u = plain.linear(a, gate).astype(np.float64), plain.linear(a, up).astype(np.float64)
    if act == 4:
        g, u = np.minimum(g, 2.0), np.clip(u, -2.0, 2.0)
        want = g / (1 + np.exp(-1.702 * g)) * (u + 1.0)
    else:
        g, u = g + bg, u + bu
        want = u * (g / (1 + np.exp(-g)) if act == 5 else 0.5 * g * (1 + np.tanh(np.sqrt(2 / np.pi) * (g + 0.044715 * g ** 3))))
    assert rel_err(host(wide[:, :I]), want) < TOL["bfloat16"]
    if ones:
        assert (wide[:, I] == 1).all() and (wide[:, I + 1:I + ones] == 0).all()
    assert (wide[:, I + ones:] == 7).all()


@pytest.mark.parametrize("M", [5, 300, 640])
def test_silu_product_and_split_sums_with_the_weight_in_k_blocks(ops, M):
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(M)
    I, K = 352, 264
    a = as_stored(rng.standard_normal((M, K)), "bfloat16")
    gate, up = as_stored(rng.standard_normal((I, K)) * 0.3, "bfloat16"), as_stored(rng.standard_normal((I, K)) * 0.3, "bfloat16")
    g = ops.bound_gemm(ops.interleave_gate_up(dev(gate, torch.bfloat16), dev(up, torch.bfloat16)), silu=True)
    assert g.packed_rows == 2 * I
    out = torch.full((M, I), float("nan"), device="cuda", dtype=torch.bfloat16)
    g(dev(a, torch.bfloat16), out)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(out), plain.swiglu(plain.linear(a, gate), plain.linear(a, up))) < TOL["bfloat16"]
    # a split product leaves its partial sums for the consumer, as with a row-major weight
    D, K2 = 520, 4096
    a2, w2 = as_stored(rng.standard_normal((M, K2)), "bfloat16"), as_stored(rng.standard_normal((D, K2)) * 0.05, "bfloat16")
    buf = {}
    got = ops.bound_gemm(dev(w2, torch.bfloat16))(dev(a2, torch.bfloat16), torch.empty(M, D, device="cuda", dtype=torch.bfloat16),
                                                  partial_scratch=lambda n: buf.setdefault("p", torch.full((n,), float("nan"), device="cuda")))
    torch.cuda.synchronize()
    gemm_select.check_status()
    if isinstance(got, ops.SplitSum):
        got = got.materialize(torch.empty(M, D, device="cuda", dtype=torch.float32))
    assert rel_err(host(got), plain.linear(a2, w2)) < TOL["bfloat16"]


def test_embedding_rows_from_a_table_in_k_blocks(ops):
    rng = np.random.default_rng(3)
    V, D = 503, 200                                      # the depth ends inside a k-block
    table = as_stored(rng.standard_normal((V, D)), "bfloat16")
    ids = np.array([0, 502, 17, 17, 256], dtype=np.int32)
    packed = ops.pack_k_blocks(dev(table, torch.bfloat16))
    assert tuple(packed.shape) == (4, V, 64) and torch.equal(ops.unpack_k_blocks(packed, D).cpu(), dev(table, torch.bfloat16).cpu())
    out = torch.full((5, D), float("nan"), device="cuda")
    ops.embed(packed, dev(ids, torch.int32), out)
    assert np.array_equal(host(out), table[ids])


@pytest.mark.parametrize("transposed,bn,splits", [(0, 16, 1), (0, 64, 1), (0, 256, 1), (1, 128, 1), (1, 256, 1), (1, 128, 3),
                                                  (1, 256, 5), (0, 128, 2)])
def test_gemm_tensor_cores_every_tiling(ops, transposed, bn, splits):
    """Every tile width, both orientations, with and without splits of k, into a strided output."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(bn + splits)
    M, N, K = 77, 300, 520
    a, w = as_stored(rng.standard_normal((M, K)), "bfloat16"), as_stored(rng.standard_normal((N, K)), "bfloat16")
    wide = torch.full((M, N + 40), 7.0, device="cuda", dtype=torch.float32)
    out = wide[:, 8:8 + N]
    gemm_select.gemm_tc(dev(a, torch.bfloat16), dev(w, torch.bfloat16), out, transposed=transposed, bn=bn, splits=splits)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(out), plain.linear(a, w)) < 2e-5
    assert (wide[:, :8] == 7).all() and (wide[:, 8 + N:] == 7).all()      # nothing is written beside the output


@pytest.mark.parametrize("bn,splits", [(128, 4), (256, 3), (256, 4)])
def test_gemm_tensor_cores_split_products_of_many_tokens(ops, bn, splits):
    """More tiles times splits than SMs: every split's CTAs walk several tiles, and the sizes end inside a tile in
    every direction. Both the finished product and the partial sums left for a consumer."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(bn + splits)
    M, N, K = 700, 2000, 1096
    a, w = as_stored(rng.standard_normal((M, K)), "bfloat16"), as_stored(rng.standard_normal((N, K)), "bfloat16")
    want = plain.linear(a, w)
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    gemm_select.gemm_tc(dev(a, torch.bfloat16), dev(w, torch.bfloat16), out, transposed=0, bn=bn, splits=splits, pair=False)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(out), want) < TOL["bfloat16"]
    scratch = torch.full((splits * M * N + 16,), float("nan"), device="cuda")
    got = gemm_select.gemm_tc(dev(a, torch.bfloat16), dev(w, torch.bfloat16), out, transposed=0, bn=bn, splits=splits, pair=False,
                              partial_scratch=lambda n: scratch[:n])
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert isinstance(got, ops.SplitSum) and got.M == M and got.N == N
    parts = scratch[:got.splits * M * N].view(got.splits, M, N)
    assert rel_err(parts.sum(0).cpu().numpy(), want) < 2e-5 and torch.isnan(scratch[got.splits * M * N:]).all()


@pytest.mark.parametrize("silu", [False, True])
def test_gemm_on_pairs_of_sms(ops, silu):
    """The cta_group::2 kernel on more tiles than there are pairs of SMs (each pair walks several,
    alternating its two accumulators), ragged in rows, columns and k, into a strided output; equal,
    bit for bit, to the one-CTA kernel, which adds the same products in the same order."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(5 + silu)
    M, N, K = 2300, 4000 + 96 * silu, 328
    a = dev(as_stored(rng.standard_normal((M, K)), "bfloat16"), torch.bfloat16)
    w = dev(as_stored(rng.standard_normal((N, K)) * 0.1, "bfloat16"), torch.bfloat16)
    cols = N // 2 if silu else N
    wide = torch.full((M, cols + 24), 7.0, device="cuda", dtype=torch.bfloat16)
    out, want = wide[:, 8:8 + cols], torch.empty(M, cols, device="cuda", dtype=torch.bfloat16)
    for _ in range(2):
        gemm_select.gemm_tc(a, w, out, silu=silu, pair=True)
    gemm_select.gemm_tc(a, w, want, silu=silu, pair=False)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert torch.equal(out, want)
    assert (wide[:, :8] == 7).all() and (wide[:, 8 + cols:] == 7).all()
    rows = slice(M - 300, M)
    ref = plain.linear(host(a)[rows], host(w))
    if silu:
        ref = ref.reshape(300, -1, 2, 16)
        ref = plain.swiglu(ref[:, :, 0].reshape(300, -1), ref[:, :, 1].reshape(300, -1))
    assert rel_err(host(out)[rows], ref) < TOL["bfloat16"]


def test_gemm_falls_back_when_tma_cannot_address_the_operands(ops):
    """K = 75 is no multiple of 8: the CUDA-core kernel serves it, same numbers."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(0)
    a, w = as_stored(rng.standard_normal((40, 75)), "bfloat16"), as_stored(rng.standard_normal((90, 75)), "bfloat16")
    ad, wd = dev(a, torch.bfloat16), dev(w, torch.bfloat16)
    out = torch.empty(40, 90, device="cuda", dtype=torch.bfloat16)
    assert not gemm_select.tc_takes(ad, wd, out)
    ops.gemm(ad, wd, out)
    assert rel_err(host(out), plain.linear(a, w)) < TOL["bfloat16"]
    from tiny_inference_engine_b200.errors import InvalidArgument
    with pytest.raises(InvalidArgument, match="multiples of 8"):
        gemm_select.gemm_tc(ad, wd, out)


@pytest.mark.parametrize("Hq,Hkv,Dh,page,window", [(8, 2, 128, 16, 0), (6, 2, 64, 16, 0), (4, 4, 64, 8, 0), (16, 1, 128, 32, 0),
                                                  (3, 1, 256, 16, 0), (8, 2, 128, 16, 100), (5, 5, 64, 4, 37), (32, 2, 64, 64, 0)])
def test_tensor_core_attention_prompt_and_decode(ops, Hq, Hkv, Dh, page, window):
    """The mma kernels on a mixed batch with scattered pages: three sequences bring portions over a
    cached prefix (one of them its whole prompt, one a portion that is no multiple of anything),
    three bring one token with one, two and twelve splits."""
    rng = np.random.default_rng(Hq * Dh + page)
    ctx = [45, 300, 130, 1, 70, 700]
    new = [45, 17, 129, 1, 1, 1]
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", ctx, Hkv, Dh, page, 128 * 16 // page)
    T = sum(new)
    stride = Hq * Dh + 2 * Hkv * Dh                     # q as the engine holds it: the first columns of the qkv rows
    qkv = as_stored(rng.standard_normal((T, stride)), "bfloat16")
    q = qkv[:, :Hq * Dh]
    qs = np.concatenate([[0], np.cumsum(new)])
    scale = 1.0 / np.sqrt(Dh)
    want = np.concatenate([dense_reference(q[qs[i]:qs[i + 1]], ks[i], vs[i], Hq, Hkv, Dh, new[i], window) for i in range(6)])
    qd = dev(qkv, torch.bfloat16)[:, :Hq * Dh]
    assert ops.attention_tc_takes(qd, Hq, Hkv, Dh)
    out = torch.full((T, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
    meta = (dev(qs, torch.int32), dev(np.array(ctx), torch.int32), dev(bt, torch.int32))
    n_multi = new[0] + new[1] + new[2]
    ops.attention_prompt_tc(qd, dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, *meta, 3, 129, Hq, Hkv, Dh, scale, window)
    assert rel_err(host(out)[:n_multi], want[:n_multi]) < TOL["bfloat16"]
    assert torch.isnan(out[n_multi:].float()).all()          # rows of other sequences are not touched
    if ops.attention_decode_tma_takes(qd, Hq, Hkv, Dh, page):
        from tiny_inference_engine_b200.ops import gemm_select
        out[:] = float("nan")
        ops.attention_prompt_tma(qd, dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, *meta, 3, 129, Hq, Hkv, Dh, scale, window)
        torch.cuda.synchronize()
        gemm_select.check_status()
        assert rel_err(host(out)[:n_multi], want[:n_multi]) < TOL["bfloat16"], "TMA-fed prompt kernel"
        assert torch.isnan(out[n_multi:].float()).all()
        if Dh in (64, 128):
            out[:] = float("nan")
            ops.attention_prompt_umma(qd, dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, *meta, 3, 129, Hq, Hkv, Dh, scale, window)
            torch.cuda.synchronize()
            gemm_select.check_status()
            assert rel_err(host(out)[:n_multi], want[:n_multi]) < TOL["bfloat16"], "tcgen05 prompt kernel"
            assert torch.isnan(out[n_multi:].float()).all()
    scratch = torch.empty(ops.attention_split_scratch_floats(3, Hq, Dh, 12), device="cuda")
    ops.attention_decode_tc(qd, dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, *meta, Hq, Hkv, Dh, scale,
                            dev(np.array([3, 4, 5]), torch.int32), 3, 64, 12, scratch, window)
    assert rel_err(host(out), want) < TOL["bfloat16"]
    # the TMA-fed decode kernel (pages that are powers of two from 8 up), with 1, 2 and many splits, twice
    # in a row so that the second launch finds the counters the first one left
    if ops.attention_decode_tma_takes(qd, Hq, Hkv, Dh, page):
        from tiny_inference_engine_b200.ops import gemm_select
        counters = torch.zeros(3 * Hkv, dtype=torch.int32, device="cuda")
        # and with the splits of a sequence as one cluster that merges through shared memory (2, 4, 8, 16 splits; one
        # of the sequences has a single key, so most of its cluster has nothing to add)
        scratch = torch.empty(ops.attention_split_scratch_floats(3, Hq, Dh, 16), device="cuda")
        for split_keys, max_splits, cluster in ((64, 12, False), (512, 2, False), (1024, 1, False), (64, 12, False), (64, 16, True),
                                                (512, 2, True), (256, 4, True), (128, 8, True), (64, 16, True)):
            out[n_multi:] = float("nan")
            ops.attention_decode_tma(qd, dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, *meta, Hq, Hkv, Dh, scale,
                                     3 if cluster else dev(np.array([3, 4, 5]), torch.int32), 3, split_keys, max_splits, scratch,
                                     counters, window, cluster=cluster)
            torch.cuda.synchronize()
            gemm_select.check_status()
            assert rel_err(host(out), want) < TOL["bfloat16"], f"split_keys={split_keys} cluster={cluster}"
            assert not counters.any()


@pytest.mark.parametrize("Hq,Hkv,Dh,page,window", [(8, 2, 128, 16, 0), (4, 4, 64, 8, 0), (16, 1, 128, 32, 0), (6, 2, 256, 16, 0),
                                                  (8, 2, 128, 16, 100), (32, 2, 64, 64, 0)])
@pytest.mark.parametrize("source", ["rows", "partial sums"])
def test_decode_attention_that_prepares_its_own_heads(ops, Hq, Hkv, Dh, page, window, source):
    """A step of single tokens, straight from the q/k/v product's output: the kernel norms and rotates its query
    heads, makes the newest key and value, stores them and uses them. Equal, bit for bit, to the q/k norm + RoPE +
    append kernel followed by the TMA-fed decode attention (outputs and both cache planes; with eight splits the
    kernel under test merges them as a cluster through shared memory, the other through scratch memory), and right against the
    plain attention over keys that include the newest. Contexts that end at the first and the last key of a tile,
    of a page and of a split, one of a single key, one empty (a sequence that pads a captured batch); the newest
    key's slot holds junk before the step, and so do the slots behind it."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(Hq + Dh + page)
    contexts = [1, 64, 65, 300, 129, 0, 257, 256]
    S = len(contexts)
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", [max(c, 1) for c in contexts], Hkv, Dh, page, 128 * 16 // page)
    width = (Hq + 2 * Hkv) * Dh
    rows = as_stored(rng.standard_normal((S, width)), "bfloat16")
    qw, kw = (1 + 0.2 * rng.standard_normal(Dh)).astype(np.float32), (1 + 0.2 * rng.standard_normal(Dh)).astype(np.float32)
    inv = plain.rope_inv_freq(1e6, Dh)
    pos = np.array([max(c - 1, 0) for c in contexts])
    slots = np.array([bt[i, pos[i] // page] * page + pos[i] % page if contexts[i] > 0 else -1 for i in range(S)])
    for i in range(S):                          # the newest key's slot, and the rest of its page, hold junk
        if contexts[i] > 0:
            kc[bt[i, pos[i] // page], :, pos[i] % page:] = 7.0
            vc[bt[i, pos[i] // page], :, pos[i] % page:] = -7.0
    qs = np.arange(S + 1)
    meta = (dev(qs, torch.int32), dev(np.array(contexts), torch.int32), dev(bt, torch.int32))
    seqs = dev(np.arange(S), torch.int32)
    scale = 1.0 / np.sqrt(Dh)
    partial = None
    if source == "partial sums":                # three float partial sums whose sum, in order, is what the kernels see
        parts = np.stack([rows * 0.5, rows * 0.25, rows * 0.25]).astype(np.float32)
        partial = ops.SplitSum(dev(parts).reshape(-1), 3, S, width)
    results = []
    for fused in (False, True):
        kcd, vcd = dev(kc, torch.bfloat16), dev(vc, torch.bfloat16)
        qkv = dev(rows if partial is None else np.zeros_like(rows), torch.bfloat16)
        out = torch.full((S, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
        scratch = torch.empty(ops.attention_split_scratch_floats(S, Hq, Dh, 8), device="cuda")
        counters = torch.zeros(S * Hkv, dtype=torch.int32, device="cuda")
        for split_keys, max_splits in ((64, 8), (128, 3), (512, 1)):
            if fused:
                assert ops.attention_decode_prep_takes(qkv, Hq, Hkv, Dh, page, dev(inv))
                # (the sequences as "S in a row from 0 on" instead of a list, for every other split size)
                ops.attention_decode_prep(qkv, dev(qw), dev(kw), 1e-6, 1e-5, dev(inv), dev(pos, torch.int32), kcd, vcd, out, *meta,
                                          Hq, Hkv, Dh, scale, 0 if split_keys != 128 else seqs, S, split_keys, max_splits, scratch,
                                          counters, window, append=True, partial=partial, cluster=max_splits in ops.CLUSTER_SPLITS)
            else:
                work = qkv.clone()
                ops.qk_norm_rope_append(work, dev(qw), dev(kw), 1e-6, 1e-5, dev(inv), dev(pos, torch.int32), dev(slots, torch.int32),
                                        kcd, vcd, Hq, Hkv, Dh, partial=partial)
                ops.attention_decode_tma(work[:, :Hq * Dh], kcd, vcd, out, *meta, Hq, Hkv, Dh, scale, seqs, S, split_keys,
                                         max_splits, scratch, counters, window)
            torch.cuda.synchronize()
            gemm_select.check_status()
            assert not counters.any()
            results.append((fused, split_keys, out.clone(), kcd.clone(), vcd.clone()))
    half = len(results) // 2
    for (_, sk, o0, k0, v0), (_, _, o1, k1, v1) in zip(results[:half], results[half:]):
        assert torch.equal(o0, o1), f"outputs differ at split_keys={sk}"
        assert torch.equal(k0, k1) and torch.equal(v0, v1), "cache planes differ"
    # against the plain formulas: the newest key and value are among the keys
    q, k, v = rows[:, :Hq * Dh], rows[:, Hq * Dh:(Hq + Hkv) * Dh], rows[:, (Hq + Hkv) * Dh:]
    want_q = as_stored(plain.rope_neox(plain.rms_norm(q.reshape(S * Hq, Dh), qw, 1e-6).reshape(S, -1), pos, Hq, Dh, 1e6), "bfloat16")
    want_k = as_stored(plain.rope_neox(plain.rms_norm(k.reshape(S * Hkv, Dh), kw, 1e-5).reshape(S, -1), pos, Hkv, Dh, 1e6), "bfloat16")
    got = host(results[-1][2])
    for i, c in enumerate(contexts):
        if c == 0:
            assert not got[i].any()
            continue
        keys = np.concatenate([ks[i][:c - 1], want_k[i].reshape(1, Hkv, Dh)])
        vals = np.concatenate([vs[i][:c - 1], v[i].reshape(1, Hkv, Dh)])
        want = dense_reference(want_q[i:i + 1], keys, vals, Hq, Hkv, Dh, 1, window)
        assert rel_err(got[i:i + 1], want) < TOL["bfloat16"], f"context {c}"
    # without the append (a layer that reads another layer's cache): the cache is read as it is and left as it is
    kcd, vcd = results[4][3].clone(), results[4][4].clone()     # the planes as the run with 3 splits of 128 keys left them
    before_k, before_v = kcd.clone(), vcd.clone()
    out = torch.full((S, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
    q_only = dev(rows, torch.bfloat16)[:, :Hq * Dh]
    ops.attention_decode_prep(q_only, dev(qw), dev(kw), 1e-6, 1e-5, dev(inv), dev(pos, torch.int32), kcd, vcd, out, *meta,
                              Hq, Hkv, Dh, scale, seqs, S, 128, 3, scratch, counters, window, append=False)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert torch.equal(kcd, before_k) and torch.equal(vcd, before_v)
    if partial is None:
        assert torch.equal(out, results[4][2])


@pytest.mark.parametrize("far", [0, 15, 16, 63, 64, 65, 255, 256, 511, 512, 1022, 1023])
def test_tensor_core_attention_finds_one_far_key(ops, far):
    """As test_one_far_key_among_a_thousand_is_found, for the mma kernels: edges of pages (16),
    of a warp's 16 keys, of 64-key tiles, of 256-key splits, the first and the last key."""
    rng = np.random.default_rng(far)
    Hq, Hkv, Dh, page, n = 8, 2, 64, 16, 1024
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", [n, n], Hkv, Dh, page, 140)
    for n_new in (1, 40):                                  # decode kernel, then the prompt kernel (last 40 rows)
        q = np.zeros((n_new, Hq * Dh), dtype=np.float32)
        for h in range(Hq):
            q[-1, h * Dh:(h + 1) * Dh] = 8.0 * ks[0][far, h // 4] * np.sqrt(Dh)
        q = as_stored(q, "bfloat16")
        want = dense_reference(q, ks[0], vs[0], Hq, Hkv, Dh, n_new)
        one_hot = np.concatenate([vs[0][far, h // 4] for h in range(Hq)])
        if far <= n - n_new or n_new == 1:
            assert np.abs(want[-1] - one_hot).max() < 2e-3
        meta = (dev(np.array([0, n_new]), torch.int32), dev(np.array([n]), torch.int32), dev(bt[:1], torch.int32))
        out = torch.zeros(n_new, Hq * Dh, device="cuda", dtype=torch.bfloat16)
        args = (dev(q, torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out)
        if n_new == 1:
            scratch = torch.empty(ops.attention_split_scratch_floats(1, Hq, Dh, 4), device="cuda")
            ops.attention_decode_tc(*args, *meta, Hq, Hkv, Dh, 1 / np.sqrt(Dh), dev(np.array([0]), torch.int32), 1, 256, 4, scratch)
            assert np.abs(host(out)[-1] - want[-1]).max() < 2e-2, "cp.async decode kernel"
            out.zero_()
            ops.attention_decode_tma(*args, *meta, Hq, Hkv, Dh, 1 / np.sqrt(Dh), dev(np.array([0]), torch.int32), 1, 256, 4,
                                     scratch, torch.zeros(Hkv, dtype=torch.int32, device="cuda"))
        else:
            ops.attention_prompt_tc(*args, *meta, 1, n_new, Hq, Hkv, Dh, 1 / np.sqrt(Dh))
            assert np.abs(host(out)[-1] - want[-1]).max() < 2e-2, "cp.async prompt kernel"
            out.zero_()
            ops.attention_prompt_tma(*args, *meta, 1, n_new, Hq, Hkv, Dh, 1 / np.sqrt(Dh))
            assert np.abs(host(out)[-1] - want[-1]).max() < 2e-2, "TMA-fed prompt kernel"
            out.zero_()
            ops.attention_prompt_umma(*args, *meta, 1, n_new, Hq, Hkv, Dh, 1 / np.sqrt(Dh))
        assert np.abs(host(out)[-1] - want[-1]).max() < 2e-2, f"n_new={n_new}"


@pytest.mark.parametrize("Hq,Hkv,Dh,page,window", [(8, 2, 128, 16, 0), (6, 2, 64, 8, 0), (3, 3, 128, 64, 0), (16, 1, 64, 128, 0),
                                                  (8, 2, 128, 16, 70), (10, 2, 64, 32, 333), (32, 2, 128, 16, 0), (32, 2, 128, 16, 100)])
def test_tcgen05_prompt_attention_on_long_portions(ops, Hq, Hkv, Dh, page, window):
    """Portions that fill several 256-row tiles and end inside one: a whole prompt, a portion over a long
    cached prefix, a portion whose rows end one short of a tile, and a short one; scattered pages. With 16 query
    heads to a key head there are so many rows that a CTA takes two row tiles; with fewer, one."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(Hq + Dh + page + window)
    ctx = [333, 900, 64 * 3 - 1, 21]
    new = [333, 257, 64 * 3 - 1, 5]
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", ctx, Hkv, Dh, page, sum(-(-c // page) for c in ctx) + 5)
    T = sum(new)
    qkv = as_stored(rng.standard_normal((T, Hq * Dh + 2 * Hkv * Dh)), "bfloat16")
    q = qkv[:, :Hq * Dh]
    qs = np.concatenate([[0], np.cumsum(new)])
    want = np.concatenate([dense_reference(q[qs[i]:qs[i + 1]], ks[i], vs[i], Hq, Hkv, Dh, new[i], window) for i in range(4)])
    qd = dev(qkv, torch.bfloat16)[:, :Hq * Dh]
    out = torch.full((T + 3, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
    meta = (dev(qs, torch.int32), dev(np.array(ctx), torch.int32), dev(bt, torch.int32))
    assert ops.attention_prompt_umma_takes(qd, Hq, Hkv, Dh, page, max(new))
    for _ in range(2):
        ops.attention_prompt_umma(qd, dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out[:T], *meta, 4, max(new), Hq, Hkv, Dh,
                                  1 / np.sqrt(Dh), window)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(out)[:T], want) < TOL["bfloat16"]
    assert torch.isnan(out[T:].float()).all()


def test_tcgen05_prompt_attention_when_the_maximum_keeps_growing(ops):
    """Scores that rise along the keys by about 3 (in powers of two) a key: every tile moves the
    reference point of the exponentials, so the accumulator in tensor memory is rescaled again and again;
    and scores that fall, so that it never is after the first tile."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(11)
    Hq, Hkv, Dh, page, n = 4, 1, 64, 16, 640
    for rising in (True, False):
        kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", [n], Hkv, Dh, page, 48)
        u = rng.standard_normal(Dh)
        u /= np.linalg.norm(u)
        ramp = np.arange(n) if rising else n - np.arange(n)
        keys = as_stored(ramp[:, None] * u[None, :] * 0.25 + 0.05 * rng.standard_normal((n, Dh)), "bfloat16")
        for t in range(n):                                  # overwrite the cached keys in their pages
            kc[bt[0, t // page], 0, t % page] = keys[t]
        q = as_stored(np.tile(u * 8.0 * np.sqrt(Dh) * np.log(2), (n, Hq)) + 0.1 * rng.standard_normal((n, Hq * Dh)), "bfloat16")
        want = dense_reference(q, keys.reshape(n, Hkv, Dh), vs[0], Hq, Hkv, Dh, n)
        out = torch.zeros(n, Hq * Dh, device="cuda", dtype=torch.bfloat16)
        ops.attention_prompt_umma(dev(q, torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out,
                                  dev(np.array([0, n]), torch.int32), dev(np.array([n]), torch.int32), dev(bt, torch.int32), 1, n,
                                  Hq, Hkv, Dh, 1 / np.sqrt(Dh))
        torch.cuda.synchronize()
        gemm_select.check_status()
        assert rel_err(host(out), want) < TOL["bfloat16"], f"rising={rising}"


@pytest.mark.parametrize("page,longest", [(8, 4500), (16, 8300)])
def test_decode_attention_over_long_contexts_with_the_longest_splits(ops, page, longest):
    """Contexts beyond what one split may hold (the kernel keeps a split's page ids in shared memory): the part's
    choice of split size stays inside the limit and the result is the dense one."""
    from tiny_inference_engine_b200.ops import gemm_select
    from tiny_inference_engine_b200.parts.attention import decode_splits
    rng = np.random.default_rng(page)
    Hq, Hkv, Dh = 4, 2, 64
    split_keys, max_splits = decode_splits(longest, 200, Hkv, page)       # so many sequences that each gets one CTA per kv head
    assert max_splits == 2 and split_keys < longest
    ctx = [longest, split_keys + 1, split_keys, 10, 1]
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", ctx, Hkv, Dh, page, sum(-(-c // page) for c in ctx) + 3)
    S = len(ctx)
    q = as_stored(rng.standard_normal((S, Hq * Dh)), "bfloat16")
    want = np.concatenate([dense_reference(q[i:i + 1], ks[i], vs[i], Hq, Hkv, Dh, 1) for i in range(S)])
    out = torch.full((S, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
    scratch = torch.empty(ops.attention_split_scratch_floats(S, Hq, Dh, max_splits), device="cuda")
    counters = torch.zeros(S * Hkv, dtype=torch.int32, device="cuda")
    ops.attention_decode_tma(dev(q, torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out,
                             dev(np.arange(S + 1), torch.int32), dev(np.array(ctx), torch.int32), dev(bt, torch.int32), Hq, Hkv, Dh,
                             1 / np.sqrt(Dh), dev(np.arange(S), torch.int32), S, split_keys, max_splits, scratch, counters)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(out), want) < TOL["bfloat16"] and not counters.any()


@pytest.mark.parametrize("split_keys", [128, 1024])
def test_decode_attention_of_more_ctas_than_places_in_any_order(ops, split_keys):
    """More CTAs than fit at once: a sequence's heads start together and the list's order says which sequences start first. Each
    sequence's output has the same bits in any order, also with the sequences as they stand, and in a launch of few CTAs."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(split_keys)
    Hq, Hkv, Dh, page = 16, 8, 64, 16
    ctx = [int(c) for c in rng.integers(1, 700, 45)]
    S, max_splits = len(ctx), -(-max(ctx) // split_keys)
    assert S * Hkv * max_splits > 2 * 148
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", ctx, Hkv, Dh, page, sum(-(-c // page) for c in ctx) + 3)
    q = as_stored(rng.standard_normal((S, Hq * Dh)), "bfloat16")
    want = np.concatenate([dense_reference(q[i:i + 1], ks[i], vs[i], Hq, Hkv, Dh, 1) for i in range(S)])
    scratch = torch.empty(ops.attention_split_scratch_floats(S, Hq, Dh, max_splits), device="cuda")
    counters = torch.zeros(S * Hkv, dtype=torch.int32, device="cuda")
    args = (dev(q, torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16))
    meta = (dev(np.arange(S + 1), torch.int32), dev(np.array(ctx), torch.int32), dev(bt, torch.int32), Hq, Hkv, Dh, 1 / np.sqrt(Dh))
    longest_first = np.argsort(-np.array(ctx), kind="stable")
    orders = [[(0, S)], [(dev(np.arange(S), torch.int32), S)], [(dev(longest_first, torch.int32), S)], [(dev(longest_first[::-1].copy(), torch.int32), S)],
              [(dev(part.copy(), torch.int32), len(part)) for part in np.array_split(longest_first, 15)]]
    outs = []
    for launches in orders:
        out = torch.full((S, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
        for seqs, n in launches:
            ops.attention_decode_tma(*args, out, *meta, seqs, n, split_keys, max_splits, scratch, counters)
        outs.append(out)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert rel_err(host(outs[0]), want) < TOL["bfloat16"] and not counters.any()
    assert all(torch.equal(outs[0], out) for out in outs[1:])


def test_a_context_beyond_the_splits_a_call_allows_costs_time_or_is_refused_but_never_keys(ops):
    """A caller of the exported kernels who sizes max_splits from something else than the longest context: the
    CUDA-core and cp.async kernels let the last split take the rest (the merge reads no more splits than there
    are), the TMA kernel, whose splits are bounded by its page table in shared memory, says so in the status word."""
    from tiny_inference_engine_b200.errors import TieError
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(77)
    Hq, Hkv, Dh, page = 4, 2, 64, 16
    ctx = [700, 130, 64, 1]                      # 700 keys need 6 splits of 128; the call allows 2
    split_keys, max_splits, S = 128, 2, len(ctx)
    for dtype in ("float32", "bfloat16"):
        kc, vc, bt, ks, vs = paged_cache(rng, dtype, ctx, Hkv, Dh, page, sum(-(-c // page) for c in ctx) + 3)
        q = as_stored(rng.standard_normal((S, Hq * Dh)), dtype)
        want = np.concatenate([dense_reference(q[i:i + 1], ks[i], vs[i], Hq, Hkv, Dh, 1) for i in range(S)])
        args = (dev(np.arange(S + 1), torch.int32), dev(np.array(ctx), torch.int32), dev(bt, torch.int32), Hq, Hkv, Dh,
                1 / np.sqrt(Dh), dev(np.arange(S), torch.int32), S, split_keys, max_splits)
        fns = [ops.attention_split] + ([ops.attention_decode_tc] if dtype == "bfloat16" else [])
        for fn in fns:
            out = torch.full((S, Hq * Dh), float("nan"), device="cuda", dtype=DT[dtype])
            scratch = torch.full((ops.attention_split_scratch_floats(S, Hq, Dh, max_splits),), float("nan"), device="cuda")
            fn(dev(q, DT[dtype]), dev(kc, DT[dtype]), dev(vc, DT[dtype]), out, *args, scratch)
            torch.cuda.synchronize()
            assert rel_err(host(out), want) < TOL[dtype], fn.__name__
    out = torch.full((S, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
    counters = torch.zeros(S * Hkv, dtype=torch.int32, device="cuda")
    ops.attention_decode_tma(dev(q, torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, *args, scratch, counters)
    torch.cuda.synchronize()
    with pytest.raises(TieError, match="fewer splits"):
        gemm_select.check_status()
    assert torch.isnan(out[0].float()).all() and rel_err(host(out)[1:], want[1:]) < TOL["bfloat16"]
    gemm_select.check_status()                   # read and cleared


def test_tensor_core_attention_refuses_other_sizes(ops):
    q = torch.zeros(4, 2 * 48, device="cuda", dtype=torch.bfloat16)
    assert not ops.attention_tc_takes(q, 2, 1, 48)
    assert not ops.attention_tc_takes(torch.zeros(4, 34 * 64, device="cuda", dtype=torch.bfloat16), 34, 2, 64)
    assert not ops.attention_tc_takes(torch.zeros(4, 128, device="cuda"), 2, 1, 64)


@pytest.mark.parametrize("M", [100, 200, 300])
def test_split_products_of_many_tokens_feed_the_norm(ops, M):
    """Between 65 and a few hundred tokens a product with few output tiles cuts k as well (128-token row
    tiles, or the weights on the 128-row side up to 128 tokens): the partial sums reach the add+norm
    kernel as they are."""
    from tiny_inference_engine_b200.ops import gemm_select
    rng = np.random.default_rng(M)
    D, K = 520, 4096
    transposed, bn, splits = gemm_select.plan(M, D, K)
    assert splits > 1 and transposed == (M <= 128)
    a, w = as_stored(rng.standard_normal((M, K)), "bfloat16"), as_stored(rng.standard_normal((D, K)) * 0.05, "bfloat16")
    buf = {}
    got = ops.gemm(dev(a, torch.bfloat16), dev(w, torch.bfloat16), torch.empty(M, D, device="cuda", dtype=torch.bfloat16),
                   partial_scratch=lambda n: buf.setdefault("p", torch.full((n,), float("nan"), device="cuda")))
    assert isinstance(got, ops.SplitSum) and 1 < got.splits <= splits and (got.M, got.N) == (M, D)
    prod = plain.linear(a, w)
    x = rng.standard_normal((M, D)).astype(np.float32)
    wn = (1 + 0.1 * rng.standard_normal(D)).astype(np.float32)
    xd, out = dev(x), torch.empty(M, D, device="cuda", dtype=torch.bfloat16)
    ops.add_rmsnorm(xd, got, dev(wn), 1e-6, out)
    torch.cuda.synchronize()
    gemm_select.check_status()
    assert np.abs(host(xd) - (x + prod)).max() < 1e-4 * np.abs(prod).max()
    assert rel_err(host(out), plain.rms_norm(x + prod, wn, 1e-6)) < TOL["bfloat16"]


def test_split_products_hand_partial_sums_to_their_consumers(ops):
    """A decode-sized product whose k range is cut leaves float partial sums; the add+norm kernel and
    the q/k norm + RoPE + append kernel add them up themselves. Same numbers as the unsplit way."""
    rng = np.random.default_rng(3)
    M, D, K = 5, 1024, 2048
    a, w = as_stored(rng.standard_normal((M, K)), "bfloat16"), as_stored(rng.standard_normal((D, K)) * 0.05, "bfloat16")
    bufs = {}
    got = ops.gemm(dev(a, torch.bfloat16), dev(w, torch.bfloat16), torch.empty(M, D, device="cuda", dtype=torch.bfloat16),
                   partial_scratch=lambda n: bufs.setdefault("p", torch.empty(n, device="cuda")))
    assert isinstance(got, ops.SplitSum) and got.splits > 1 and (got.M, got.N) == (M, D)
    prod = plain.linear(a, w)
    whole = got.materialize(torch.empty(M, D, device="cuda"))
    assert rel_err(host(whole), prod) < 2e-5
    # residual add + norm straight from the partial sums
    x = rng.standard_normal((M, D)).astype(np.float32)
    wn = (1 + 0.1 * rng.standard_normal(D)).astype(np.float32)
    xd, out = dev(x), torch.empty(M, D, device="cuda", dtype=torch.bfloat16)
    ops.add_rmsnorm(xd, got, dev(wn), 1e-6, out)
    assert np.abs(host(xd) - (x + prod)).max() < 1e-4 * np.abs(prod).max()
    assert rel_err(host(out), plain.rms_norm(x + prod, wn, 1e-6)) < TOL["bfloat16"]
    rows = np.array([4, 1])
    out2, x2 = torch.empty(2, D, device="cuda", dtype=torch.bfloat16), dev(x)
    ops.add_rmsnorm(x2, got, dev(wn), 1e-6, out2, rows=dev(rows, torch.int32))
    assert np.array_equal(host(x2), x) and rel_err(host(out2), plain.rms_norm((x + prod)[rows], wn, 1e-6)) < TOL["bfloat16"]
    # q/k norm + RoPE + append from the partial sums of a q,k,v product
    Hq, Hkv, Dh, page = 4, 2, 128, 16
    width = (Hq + 2 * Hkv) * Dh
    wq = as_stored(rng.standard_normal((width, K)) * 0.05, "bfloat16")
    qkv = torch.zeros(M, width, device="cuda", dtype=torch.bfloat16)
    ps = ops.gemm(dev(a, torch.bfloat16), dev(wq, torch.bfloat16), qkv,
                  partial_scratch=lambda n: bufs.setdefault("q", torch.empty(n, device="cuda")))
    assert isinstance(ps, ops.SplitSum)
    full = plain.linear(a, wq)
    qw, kw = (1 + 0.2 * rng.standard_normal(Dh)).astype(np.float32), (1 + 0.2 * rng.standard_normal(Dh)).astype(np.float32)
    pos, slots = np.array([0, 5, 77, 1000, 3]), np.array([3, 17, 40, -1, 8])
    kc, vc = torch.zeros(4, Hkv, page, Dh, device="cuda", dtype=torch.bfloat16), torch.zeros(4, Hkv, page, Dh, device="cuda", dtype=torch.bfloat16)
    ops.qk_norm_rope_append(qkv, dev(qw), dev(kw), 1e-6, 1e-6, dev(plain.rope_inv_freq(1e6, Dh)), dev(pos, torch.int32),
                            dev(slots, torch.int32), kc, vc, Hq, Hkv, Dh, partial=ps)
    q, k, v = full[:, :Hq * Dh], full[:, Hq * Dh:(Hq + Hkv) * Dh], full[:, (Hq + Hkv) * Dh:]
    want_q = plain.rope_neox(plain.rms_norm(q.reshape(M * Hq, Dh), qw, 1e-6).reshape(M, -1), pos, Hq, Dh, 1e6)
    want_k = plain.rope_neox(plain.rms_norm(k.reshape(M * Hkv, Dh), kw, 1e-6).reshape(M, -1), pos, Hkv, Dh, 1e6)
    assert rel_err(host(qkv)[:, :Hq * Dh], want_q) < TOL["bfloat16"]
    for t in range(M):
        if slots[t] >= 0:
            p, o = slots[t] // page, slots[t] % page
            assert rel_err(host(kc)[p, :, o].reshape(1, -1), want_k[t].reshape(1, -1)) < TOL["bfloat16"]
            assert rel_err(host(vc)[p, :, o].reshape(1, -1), v[t].reshape(1, -1)) < TOL["bfloat16"]


@pytest.mark.parametrize("M", [1, 7, 64, 200, 300, 700])
@pytest.mark.parametrize("I,K", [(16, 64), (48, 72), (208, 136), (1536, 1024)])
def test_gemm_with_silu_epilogue(ops, M, I, K):
    """silu(a gate^T) * (a up^T) in the product's epilogue, both tilings, widths that end inside a tile."""
    rng = np.random.default_rng(M + I)
    a = as_stored(rng.standard_normal((M, K)), "bfloat16")
    gate, up = as_stored(rng.standard_normal((I, K)) * 0.2, "bfloat16"), as_stored(rng.standard_normal((I, K)) * 0.2, "bfloat16")
    w = ops.interleave_gate_up(dev(gate, torch.bfloat16), dev(up, torch.bfloat16))
    assert np.array_equal(host(w)[:16], gate[:16]) and np.array_equal(host(w)[16:32], up[:16])
    out = torch.full((M, I), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_silu(dev(a, torch.bfloat16), w, out)
    assert rel_err(host(out), plain.swiglu(plain.linear(a, gate), plain.linear(a, up))) < TOL["bfloat16"]


@pytest.mark.parametrize("mode", ["delta", "channel", "head"])
@pytest.mark.parametrize("H,G,dim,vdim,lens", [(2, 2, 128, 128, [1, 16, 33]), (4, 2, 64, 64, [15, 17]), (3, 3, 128, 20, [50])])
def test_recurrence_in_chunks(ops, mode, H, G, dim, vdim, lens, monkeypatch):
    """The three recurrences sixteen tokens at a time against the plain loop in float64: chunks that end in the middle, single tokens, value
    heads that fill no block of columns, decays down to zero; the convolution's inputs as the kernel that walks token by token leaves them;
    and a token with a NaN leaves the tokens ahead of it in its chunk, and the other sequences, as they are."""
    from types import SimpleNamespace
    from tiny_inference_engine_b200.engine.workspace import Workspace
    if mode == "channel":
        G = H
    rng = np.random.default_rng(H * dim + vdim + len(lens))
    T, per, taps = sum(lens), H // G, 4
    q, k = rng.standard_normal((T, G, dim)), rng.standard_normal((T, G, dim))
    q, k = q / np.linalg.norm(q, axis=-1, keepdims=True), k / np.linalg.norm(k, axis=-1, keepdims=True)
    v = rng.standard_normal((T, H, vdim))
    beta = rng.uniform(0.1, 1.0, (T, H)) if mode != "channel" else None
    decay = rng.uniform(0.3, 1.0, (T, H) if mode == "head" else (T, H, dim))
    decay.reshape(T, H, -1)[T // 2] = 0.0                      # a token that forgets everything
    S0 = rng.standard_normal((len(lens), H, dim, vdim))
    C = 2 * G * dim + H * vdim
    qs = np.concatenate([[0], np.cumsum(lens)])

    def plain_loop(v):
        out, S = np.zeros((T, H, vdim)), S0.copy()
        for s, n in enumerate(lens):
            for t in range(qs[s], qs[s] + n):
                for h in range(H):
                    S[s, h] *= decay[t, h] if mode == "head" else decay[t, h][:, None]
                    u = v[t, h] * (1.0 if beta is None else beta[t, h])
                    if mode == "delta":
                        u = u - beta[t, h] * (S[s, h].T @ k[t, h // per])
                    S[s, h] += np.outer(k[t, h // per], u)
                    out[t, h] = S[s, h].T @ q[t, h // per]
        return out, S

    proj = dev(rng.standard_normal((T, C)), torch.bfloat16)
    state0 = dev(np.concatenate([S0.reshape(len(lens), -1), rng.standard_normal((len(lens), (taps - 1) * C))], axis=1))

    def engine(v, chunked):
        rows = [dev(x.reshape(T, -1)) for x in (q, k, v)]
        state, out = state0.clone(), torch.empty(T, H * vdim, device="cuda")
        monkeypatch.setattr(ops, "chunks_pay", lambda *a: chunked)
        ctx = SimpleNamespace(ws=Workspace(T, "cuda"), multi_max_queries=max(lens), max_seqs=len(lens))
        ops.delta_rule(*rows, None if beta is None else dev(beta), dev(decay.reshape(T, -1)), state, H * dim * vdim, proj, 0, G * dim, 2 * G * dim,
                       dev(qs, torch.int32), dev(np.arange(len(lens)), torch.int32), len(lens), H, G, dim, vdim, taps, out, plain=mode != "delta",
                       decay_per_head=mode == "head", chunks=ops.RecurrenceChunks(ctx))
        return host(out), host(state)

    want, S = plain_loop(v)
    out, state = engine(v, True)
    _, by_token = engine(v, False)
    assert rel_err(out, want.reshape(T, -1)) < TOL["float32"]
    assert rel_err(state[:, :H * dim * vdim], S.reshape(len(lens), -1)) < TOL["float32"]
    assert np.array_equal(state[:, H * dim * vdim:], by_token[:, H * dim * vdim:])
    sick = T - 2
    v = v.copy()
    v[sick] = np.nan
    out, _ = engine(v, True)
    assert rel_err(out[:sick], want.reshape(T, -1)[:sick]) < TOL["float32"] and np.isnan(out[sick:]).all()


def softmax_reference(q, k, v, scale, window, sink, start):
    """q [n, H, d], k [m, G, d], v [m, G, e] in float64; row i sits at start + i. Returns [n, H, e]."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    far = (start + np.arange(n))[:, None] - np.arange(k.shape[0])[None, :]
    seen = (far >= 0) & ((far < window) if window else (far >= 0))
    out = np.zeros((n, H, v.shape[2]))
    for h in range(H):
        z = np.where(seen, scale * (q[:, h] @ k[:, h // (H // G)].T), -np.inf)
        top = z.max(-1, keepdims=True) if sink is None else np.maximum(z.max(-1, keepdims=True), sink[h])
        e = np.exp(z - top)
        total = e.sum(-1, keepdims=True) + (0.0 if sink is None else np.exp(sink[h] - top))
        out[:, h] = (e / total) @ v[:, h // (H // G)]
    return out


@pytest.mark.parametrize("Dh", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,page,window,new,ctx,sinks", [
    (4, 2, 16, 0, [129, 64], [129, 400], False), (3, 3, 64, 100, [300], [333], True), (8, 1, 8, 0, [33, 2, 17], [33, 65, 700], True),
    (2, 2, 16, 0, [513], [513], False)])
def test_exact_prompt_attention_on_tcgen05(ops, Dh, Hq, Hkv, page, window, new, ctx, sinks):
    """Rows and keys that end inside tiles, portions behind cached keys, windows, sinks, one and two row tiles a CTA; weights in two
    bfloat16 terms, so the rounding of the output is what is left of the error."""
    rng = np.random.default_rng(Hq * Dh + sum(ctx))
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", ctx, Hkv, Dh, page, 90 * 16 // page + 8)
    T, qs = sum(new), np.concatenate([[0], np.cumsum(new)])
    q = as_stored(rng.standard_normal((T, Hq * Dh)) * 2, "bfloat16")
    sink = rng.uniform(-2, 6, Hq).astype(np.float32) if sinks else None
    out = torch.full((T, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.attention_prompt_exact(dev(q, torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, dev(qs, torch.int32),
                               dev(np.array(ctx), torch.int32), dev(bt, torch.int32), len(new), max(new), Hq, Hkv, Dh, Dh ** -0.5, window,
                               None if sink is None else dev(sink))
    want = np.concatenate([softmax_reference(q[qs[i]:qs[i + 1]].reshape(-1, Hq, Dh).astype(np.float64), ks[i].astype(np.float64),
                                             vs[i].astype(np.float64), Dh ** -0.5, window, sink, ctx[i] - new[i]) for i in range(len(new))])
    assert rel_err(host(out), want.reshape(T, -1)) < TOL["bfloat16"]
    # 2-norm: one rounding to bfloat16 is 2^-9 / sqrt(3) = 1.1e-3 of a value at most; weights in one term would add 1.1e-3 of their own
    assert np.linalg.norm(host(out) - want.reshape(T, -1)) < 2.0e-3 * np.linalg.norm(want)


@pytest.mark.parametrize("H,page,window,new,ctx,sinks", [(2, 16, 0, [200, 65], [200, 65], True), (3, 8, 90, [130, 64], [260, 321], False),
                                                         (1, 64, 0, [300], [450], True)])
def test_latent_attention_over_expanded_keys(ops, H, page, window, new, ctx, sinks):
    """Gathered latents (each sequence padded to whole tiles with zeros), and attention over keys and values per head beside a rotated part that all
    heads share."""
    rng = np.random.default_rng(H + sum(ctx))
    rank, kd = 64, 128
    kc, _, bt, ks, _ = paged_cache(rng, "bfloat16", ctx, 1, kd, page, 60 * 16 // page + 8)
    T, qs = sum(new), np.concatenate([[0], np.cumsum(new)])
    index = (dev(qs, torch.int32), dev(np.array(ctx), torch.int32))
    rows = ops.latent_expanded_rows(ctx, new, window)
    latents = torch.full((rows, kd), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.latent_gather(dev(kc, torch.bfloat16), *index, dev(bt, torch.int32), len(new), window, latents)
    firsts = [max(0, c - n - window + 1) // 64 * 64 if window else 0 for c, n in zip(ctx, new)]
    edges = [max(0, c - n - window + 1) if window else 0 for c, n in zip(ctx, new)]      # ahead of the first key seen: zeros too
    want_rows = np.concatenate([np.concatenate([np.zeros((e - f, kd)), k[e:, 0], np.zeros((-(len(k) - f) % 64, kd))])
                                for k, f, e in zip(ks, firsts, edges)])
    assert np.array_equal(host(latents), want_rows)
    kv = as_stored(rng.standard_normal((rows, H * 256)), "bfloat16")
    q = as_stored(rng.standard_normal((T, H * 192)) * 1.5, "bfloat16")
    sink = rng.uniform(-2, 6, H).astype(np.float32) if sinks else None
    out = torch.full((T, H * 128), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.attention_latent_expanded(dev(q, torch.bfloat16), latents, dev(kv, torch.bfloat16), out, *index, len(new), max(new), H, 192 ** -0.5, window,
                                  None if sink is None else dev(sink))
    want, base = [], 0
    for i, (n, c) in enumerate(zip(new, ctx)):
        m = c - firsts[i]
        k = np.concatenate([kv[base:base + m, :H * 128].reshape(m, H, 128), np.repeat(want_rows[base:base + m, None, rank:], H, axis=1)], axis=-1)
        v = kv[base:base + m, H * 128:].reshape(m, H, 128)
        want.append(softmax_reference(q[qs[i]:qs[i + 1]].reshape(n, H, 192).astype(np.float64), k.astype(np.float64), v.astype(np.float64), 192 ** -0.5,
                                      window, sink, c - n - firsts[i]))
        base += -(-m // 64) * 64
    want = np.concatenate(want).reshape(T, -1)
    assert np.linalg.norm(host(out) - want) < 2.0e-3 * np.linalg.norm(want)


@pytest.mark.parametrize("Dh", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,page,window,new,ctx", [
    (4, 2, 16, 0, [130], [2600]), (8, 2, 16, 0, [300, 3], [2351, 40]), (4, 4, 64, 700, [700], [1500]), (32, 8, 8, 0, [260], [2119])])
def test_keys_shared_out_over_a_cluster(ops, Dh, Hq, Hkv, page, window, new, ctx):
    """Few rows behind many keys: two and four CTAs share out the key tiles of 256 rows; a short sequence beside the long one leaves CTAs without
    keys, the last rows of a portion leave row tiles without any."""
    rng = np.random.default_rng(Hq * Dh + sum(ctx))
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", ctx, Hkv, Dh, page, 180 * 16 // page + 8)
    T, qs = sum(new), np.concatenate([[0], np.cumsum(new)])
    q = as_stored(rng.standard_normal((T, Hq * Dh)) * 2, "bfloat16")
    out = torch.full((T, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.attention_prompt_umma(dev(q, torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, dev(qs, torch.int32),
                              dev(np.array(ctx), torch.int32), dev(bt, torch.int32), len(new), max(new), Hq, Hkv, Dh, Dh ** -0.5, window,
                              max_keys=4096)
    want = np.concatenate([softmax_reference(q[qs[i]:qs[i + 1]].reshape(-1, Hq, Dh).astype(np.float64), ks[i].astype(np.float64),
                                             vs[i].astype(np.float64), Dh ** -0.5, window, None, ctx[i] - new[i]) for i in range(len(new))])
    assert rel_err(host(out), want.reshape(T, -1)) < TOL["bfloat16"]


@pytest.mark.parametrize("Dh", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,new,ctx", [(4, 2, 130, 2600), (64, 8, 150, 2900)])
@pytest.mark.parametrize("sick", ["query", "key", "value", "value of no weight", "infinite"])
def test_what_is_not_a_number_survives_shared_out_keys(ops, Dh, Hq, Hkv, new, ctx, sick):
    """Four and two CTAs a tile. A NaN in a query row, a key, a value (one whose share of the keys has a factor of zero as well) or an infinite
    score shows in the rows that see it as it does when one CTA goes through all keys, and every other row stays as it was."""
    rng = np.random.default_rng(Hq * Dh + ctx)
    page = 16
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", [ctx], Hkv, Dh, page, 180 * 16 // page + 8)
    q = rng.standard_normal((new, Hq * Dh)) * 2
    at = ctx - new + 40                                    # a key that rows 40 and up see
    rows = np.zeros((new, Hq), bool)
    if sick == "value of no weight":
        q *= 64                                            # scores of hundreds, but for the first half of the keys and a little more
        for p in range((ctx // 2 + 64) // page):
            kc[bt[0, p]] *= 0.01
            ks[0][p * page:(p + 1) * page] *= 0.01
    if sick == "query":
        q[5, 3 * Dh + 1] = np.nan
        rows[5, 3] = True
    elif sick == "infinite":
        q[5, 3 * Dh + 1], rows[5, 3] = np.inf, True        # scores of both infinities
    elif sick == "key":
        kc[bt[0, at // page], 1, at % page, 2] = np.nan
        rows[40:, Hq // Hkv:2 * Hq // Hkv] = True
    else:
        where = at if sick == "value" else 5
        vc[bt[0, where // page], 1, where % page] = np.nan
        rows[40 if sick == "value" else 0:, Hq // Hkv:2 * Hq // Hkv] = True
    args = (dev(as_stored(q, "bfloat16"), torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16))
    index = (dev(np.array([0, new]), torch.int32), dev(np.array([ctx]), torch.int32), dev(bt, torch.int32), 1, new, Hq, Hkv, Dh, Dh ** -0.5, 0)
    got = []
    for max_keys in (0, ctx):
        out = torch.full((new, Hq * Dh), 7.0, device="cuda", dtype=torch.bfloat16)
        ops.attention_prompt_umma(*args, out, *index, max_keys=max_keys)
        got.append(host(out).reshape(new, Hq, Dh))
    for out in got:
        assert np.isnan(out[rows]).all()
    # a tile's masked values are multiplied with weights of zero, so rows that do not see a sick value may be lost with either
    clean = ~np.isnan(got[0]).any(-1)
    assert clean.sum() > 0 and (sick.startswith("value") or np.array_equal(clean, ~rows))
    assert np.isfinite(got[1][clean]).all()
    want = softmax_reference(as_stored(np.nan_to_num(q, posinf=0.0), "bfloat16").reshape(-1, Hq, Dh).astype(np.float64),
                             ks[0].astype(np.float64), vs[0].astype(np.float64), Dh ** -0.5, 0, None, ctx - new)
    assert rel_err(got[1][clean], want[clean]) < TOL["bfloat16"]


@pytest.mark.parametrize("page,window,new,ctx", [(16, 100, [70, 64], [300, 513]), (8, 90, [64], [1000]), (64, 40, [65], [300])])
def test_pages_behind_a_window_are_not_gathered(ops, page, window, new, ctx):
    """Pages below a window have been given back: the table names page 0 there, which is another request's by then. Tiles begin below the
    window's first key, so NaN in page 0 must not reach the rows gathered, nor the attention over them."""
    rng = np.random.default_rng(page + window)
    H, kd = 2, 128
    kc, _, bt, ks, _ = paged_cache(rng, "bfloat16", ctx, 1, kd, page, 100 * 16 // page + 8)
    kc = np.concatenate([np.full_like(kc[:1], np.nan), kc])        # page 0: someone else's
    bt = bt + 1
    edges = [c - n - window + 1 for c, n in zip(ctx, new)]           # first key that the sequence's first row sees
    for s, edge in enumerate(edges):
        bt[s, :edge // page] = 0
        bt[s, -(-ctx[s] // page):] = 0
    qs = np.concatenate([[0], np.cumsum(new)])
    index = (dev(qs, torch.int32), dev(np.array(ctx), torch.int32))
    rows = ops.latent_expanded_rows(ctx, new, window)
    latents = torch.full((rows, kd), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.latent_gather(dev(kc, torch.bfloat16), *index, dev(bt, torch.int32), len(new), window, latents)
    want = [np.zeros((0, kd))]
    for k, c, edge in zip(ks, ctx, edges):
        first = edge // 64 * 64
        want += [np.zeros((edge - first, kd)), k[edge:, 0], np.zeros((-(c - first) % 64, kd))]
    assert np.array_equal(host(latents), np.concatenate(want))
    q = dev(as_stored(rng.standard_normal((sum(new), H * 192)), "bfloat16"), torch.bfloat16)
    out = torch.full((sum(new), H * 128), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.attention_latent_expanded(q, latents, latents.repeat(1, H * 256 // kd), out, *index, len(new), max(new), H, 192 ** -0.5, window)
    assert torch.isfinite(out.float()).all()


def test_rows_behind_the_last_query_end(ops):
    """More rows than the sequences' queries: each takes the place that its number says, as in the kernel without tiles, and the walk over a tile's
    sequences ends."""
    Hq, Hkv, Dh, page, ctx, queries, T = 2, 1, 64, 16, 20, 16, 20
    rng = np.random.default_rng(3)
    kc, vc, bt, ks, vs = paged_cache(rng, "float32", [ctx + T - queries], Hkv, Dh, page, 8)
    q = rng.standard_normal((T, Hq * Dh)).astype(np.float32)
    out = torch.full((T, Hq * Dh), float("nan"), device="cuda")
    ops.attention_rows(dev(q), dev(kc), dev(vc), out, dev(np.zeros(T), torch.int32), dev(np.array([0, queries]), torch.int32),
                       dev(np.array([ctx]), torch.int32), dev(bt, torch.int32), Hq, Hkv, Dh, Dh ** -0.5)
    assert rel_err(host(out), dense_reference(q, ks[0], vs[0], Hq, Hkv, Dh, T)) < TOL["float32"]


@pytest.mark.parametrize("Dh,new,ctx", [(32, 20, 20), (64, 40, 100), (128, 33, 64)])
def test_a_value_that_is_not_a_number_counts_at_any_weight(ops, Dh, new, ctx):
    """Key 0 scores 200 below the others, so its weight is zero in float32; its value is NaN and every row sees it. (One tile of keys and
    several, the last one seen in part.)"""
    u = np.ones(Dh, np.float32)
    page = 16
    kc, vc, bt, ks, vs = paged_cache(np.random.default_rng(1), "float32", [ctx], 1, Dh, page, 12)
    for j in range(ctx):
        kc[bt[0, j // page], 0, j % page] = (-u if j == 0 else u) * 100 / Dh
    vc[bt[0, 0], 0, 0] = np.nan
    out = torch.zeros((new, Dh), device="cuda")
    ops.attention_rows(dev(np.tile(u, (new, 1))), dev(kc), dev(vc), out, dev(np.zeros(new), torch.int32), dev(np.array([0, new]), torch.int32),
                       dev(np.array([ctx]), torch.int32), dev(bt, torch.int32), 1, 1, Dh, 1.0)
    assert np.isnan(host(out)).all()


def test_short_portions_do_not_share_tiles(ops):
    """Twenty portions of two or three tokens: a tile of 16 rows would go through the keys of eight of them one after the other, so they run
    row by row as a portion alone does, to the last bit."""
    Hq, Hkv, Dh, page = 4, 2, 64, 16
    rng = np.random.default_rng(5)
    new, ctx = [2 + i % 2 for i in range(20)], [90 + 7 * i for i in range(20)]
    kc, vc, bt, ks, vs = paged_cache(rng, "float32", ctx, Hkv, Dh, page, 330)
    qs = np.concatenate([[0], np.cumsum(new)])
    q = dev(rng.standard_normal((sum(new), Hq * Dh)))
    planes, heads = (dev(kc), dev(vc)), (Hq, Hkv, Dh, Dh ** -0.5)

    def rows(lo, hi):
        out = torch.empty((qs[hi] - qs[lo], Hq * Dh), device="cuda")
        ops.attention_rows(q[qs[lo]:qs[hi]], *planes, out, dev(np.repeat(np.arange(hi - lo), new[lo:hi]), torch.int32), dev(qs[lo:hi + 1] - qs[lo], torch.int32),
                           dev(np.array(ctx[lo:hi]), torch.int32), dev(bt[lo:hi], torch.int32), *heads)
        return out
    assert torch.equal(rows(0, 20), torch.cat([rows(i, i + 1) for i in range(20)]))


@pytest.mark.parametrize("mode", ["delta", "channel", "head"])
def test_sequences_without_tokens_keep_their_state(ops, mode, monkeypatch):
    """A step in chunks in which the first, a middle and the last sequence bring nothing: their rows of the state stay to the last bit, and the
    others' outputs are those of the walk token by token."""
    from types import SimpleNamespace
    from tiny_inference_engine_b200.engine.workspace import Workspace
    H, dim, vdim, lens, taps = 2, 64, 64, [0, 100, 0, 33, 0], 4
    rng = np.random.default_rng(4)
    T, C = sum(lens), 2 * H * dim + H * vdim
    q, k = (x / np.linalg.norm(x, axis=-1, keepdims=True) for x in rng.standard_normal((2, T, H, dim)))
    v, beta = rng.standard_normal((T, H * vdim)), rng.uniform(0.1, 1.0, (T, H)) if mode != "channel" else None
    decay = rng.uniform(0.3, 1.0, (T, H if mode == "head" else H * dim))
    state0, proj = dev(rng.standard_normal((len(lens), H * dim * vdim + (taps - 1) * C))), dev(rng.standard_normal((T, C)))
    qs = dev(np.concatenate([[0], np.cumsum(lens)]), torch.int32)
    got = {}
    for chunked in (True, False):
        monkeypatch.setattr(ops, "chunks_pay", lambda *a: chunked)
        rows = [dev(x.reshape(T, -1)) for x in (q, k, v)]
        state, out = state0.clone(), torch.empty(T, H * vdim, device="cuda")
        ctx = SimpleNamespace(ws=Workspace(T, "cuda"), multi_max_queries=max(lens), max_seqs=len(lens))
        ops.delta_rule(*rows, None if beta is None else dev(beta), dev(decay), state, H * dim * vdim, proj, 0, H * dim, 2 * H * dim, qs,
                       dev(np.arange(len(lens)), torch.int32), len(lens), H, H, dim, vdim, taps, out, plain=mode != "delta",
                       decay_per_head=mode == "head", chunks=ops.RecurrenceChunks(ctx))
        got[chunked] = host(out), host(state)
    for s, n in enumerate(lens):
        if n == 0:
            assert np.array_equal(got[True][1][s, :H * dim * vdim], host(state0)[s, :H * dim * vdim])
    assert rel_err(got[True][0], got[False][0]) < TOL["float32"] and rel_err(got[True][1], got[False][1]) < TOL["float32"]


@pytest.mark.parametrize("M,N", [(17, 65535 * 64 + 65), (65535 * 64 + 65, 17)])
def test_float_products_of_more_tiles_than_a_grid_has_in_one_direction(ops, M, N):
    """Above 65,535 tiles of columns or of rows; k of 4, so that every output can be looked at."""
    g = torch.Generator("cuda").manual_seed(M)
    a, w = torch.randn(M, 4, generator=g, device="cuda"), torch.randn(N, 4, generator=g, device="cuda")
    out = torch.full((M, N), float("nan"), device="cuda")
    ops.gemm_simt(a, w, out)
    want = sum(a[:, i:i + 1] * w[:, i] for i in range(4))
    assert (out - want).abs().max() <= 8 * 2.0 ** -24 * 4 * want.abs().max()      # four products, each rounded, in another order


def test_refused_sizes_take_no_scratch_for_chunks(ops):
    """Heads that the chunked kernels do not take, in a step that would pay: nothing is allocated for them."""
    from types import SimpleNamespace
    from tiny_inference_engine_b200.engine.workspace import Workspace
    H, dim, T = 2, 32, 400
    ctx = SimpleNamespace(ws=Workspace(T, "cuda"), multi_max_queries=T, max_seqs=1)
    rows = [torch.randn(T, H * dim, device="cuda") for _ in range(3)]
    state, out = torch.zeros(1, H * dim * dim + 9 * H * dim, device="cuda"), torch.full((T, H * dim), float("nan"), device="cuda")
    ops.delta_rule(*rows, torch.rand(T, H, device="cuda"), torch.rand(T, H * dim, device="cuda"), state, H * dim * dim, torch.randn(T, 3 * H * dim, device="cuda"),
                   0, H * dim, 2 * H * dim, torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), 1, H, H, dim,
                   dim, 4, out, chunks=ops.RecurrenceChunks(ctx))
    assert ctx.ws.bytes() == 0 and not torch.isnan(out).all()


@pytest.mark.parametrize("Dh", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,page,window,new,ctx", [
    (4, 2, 16, 1900, [300], [3000]), (32, 8, 64, 2000, [150, 49], [2900, 2100]), (4, 4, 8, 1950, [100, 2], [2049, 90]), (16, 8, 16, 1500, [600], [4000])])
def test_windows_of_keys_shared_out_over_a_cluster(ops, Dh, Hq, Hkv, page, window, new, ctx):
    """Windows long enough for four and two shares: each row tile's first key tile is clipped to a share, and a share may hold tiles of one
    row tile alone, or none (the last row tile of a portion, a short sequence beside a long one)."""
    rng = np.random.default_rng(Hq * Dh + sum(ctx))
    tiles = -(-max(new) * (Hq // Hkv) // 256) * Hkv * len(new)
    assert tiles * 2 <= 148 and window + max(new) >= 2049            # what the launcher looks at
    kc, vc, bt, ks, vs = paged_cache(rng, "bfloat16", ctx, Hkv, Dh, page, 330 * 16 // page + 8)
    T, qs = sum(new), np.concatenate([[0], np.cumsum(new)])
    q = as_stored(rng.standard_normal((T, Hq * Dh)) * 2, "bfloat16")
    want = np.concatenate([softmax_reference(q[qs[i]:qs[i + 1]].reshape(-1, Hq, Dh).astype(np.float64), ks[i].astype(np.float64),
                                             vs[i].astype(np.float64), Dh ** -0.5, window, None, ctx[i] - new[i]) for i in range(len(new))])
    got = []
    for max_keys in (0, max(ctx)):
        out = torch.full((T, Hq * Dh), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.attention_prompt_umma(dev(q, torch.bfloat16), dev(kc, torch.bfloat16), dev(vc, torch.bfloat16), out, dev(qs, torch.int32),
                                  dev(np.array(ctx), torch.int32), dev(bt, torch.int32), len(new), max(new), Hq, Hkv, Dh, Dh ** -0.5, window, max_keys=max_keys)
        got.append(host(out))
        assert rel_err(got[-1], want.reshape(T, -1)) < TOL["bfloat16"]
    assert not np.array_equal(*got)                                  # (another order of sums: the keys were shared out)


@pytest.mark.parametrize("per_head", [True, False])
def test_what_a_recurrence_in_chunks_overwrites(ops, per_head, monkeypatch):
    """One decay a head: q, k, v and the decays stay to the last bit (a state-space layer reads its values again, constant decays are a model's own tensor
    read with a stride of zero). A decay a channel: q and k are the kernels' to change, v and the decays stay."""
    from types import SimpleNamespace
    from tiny_inference_engine_b200.engine.workspace import Workspace
    H, dim, T, taps = 2, 64, 200, 4
    monkeypatch.setattr(ops, "chunks_pay", lambda *a: True)
    g = torch.Generator("cuda").manual_seed(2)
    q, k, v = (torch.randn(T, H * dim, generator=g, device="cuda") / 8 for _ in range(3))
    decay = torch.rand(H, generator=g, device="cuda").expand(T, H) if per_head else torch.rand(T, H * dim, generator=g, device="cuda")
    before = [x.clone() for x in (q, k, v, decay)]
    state, out = torch.zeros(1, H * dim * dim + (taps - 1) * 3 * H * dim, device="cuda"), torch.empty(T, H * dim, device="cuda")
    ctx = SimpleNamespace(ws=Workspace(T, "cuda"), multi_max_queries=T, max_seqs=1)
    ops.delta_rule(q, k, v, None, decay, state, H * dim * dim, torch.randn(T, 3 * H * dim, generator=g, device="cuda"), 0, H * dim, 2 * H * dim,
                   torch.tensor([0, T], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), 1, H, H, dim, dim, taps, out,
                   plain=True, decay_per_head=per_head, chunks=ops.RecurrenceChunks(ctx))
    assert ctx.ws.bytes() > 0
    same = [torch.equal(x, y) for x, y in zip((q, k, v, decay), before)]
    assert same == ([True] * 4 if per_head else [False, False, True, True])
