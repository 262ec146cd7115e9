"""Each CUDA kernel alone against its plain reference, at sizes other than the engine's."""

import math

import numpy as np
import pytest
import torch

import plain_qwen3 as plain

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


def tol(dtype):
    return dict(atol=1e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)


@pytest.fixture(scope="module")
def ops():
    from atomserve_b200 import ops

    ops.require_device()
    return ops


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [48, 100, 4096])
def test_embedding(ops, dtype, width):
    table = torch.randn(331, width, device="cuda").to(dtype)
    ids = torch.tensor([0, 330, 7, 7, 19], dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = ops.embedding(ids, table, status)
    assert torch.equal(out, table[ids.long()])
    assert int(status) == 0
    bad = torch.tensor([3, 331], dtype=torch.int32, device="cuda")
    out = ops.embedding(bad, table, status)
    assert int(status) == 1 and torch.equal(out[1], torch.zeros_like(out[1]))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,width,eps", [(1, 16, 1e-6), (7, 100, 1e-5), (33, 4096, 1e-6), (3, 5120, 3e-6)])
def test_rms_norm(ops, dtype, rows, width, eps):
    x = (torch.randn(rows, width, device="cuda") * 3).to(dtype)
    gain = 1 + 0.1 * torch.randn(width, device="cuda")
    ref = plain.rms_norm(x.float().cpu(), gain.cpu(), eps)
    out = ops.rms_norm(x, gain, eps)
    assert torch.allclose(out.float().cpu(), ref, **tol(dtype))
    pick = torch.tensor([rows - 1, 0], dtype=torch.int32, device="cuda")
    out = ops.rms_norm(x, gain, eps, pick)
    assert torch.allclose(out.float().cpu(), ref[[rows - 1, 0]], **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,inter", [(1, 24), (7, 176), (300, 12288)])
def test_silu_mul(ops, dtype, rows, inter):
    gu = (torch.randn(rows, 2 * inter, device="cuda") * 2).to(dtype)
    g, u = gu.float().cpu()[:, :inter], gu.float().cpu()[:, inter:]
    ref = g / (1 + torch.exp(-g)) * u
    assert torch.allclose(ops.silu_mul(gu).float().cpu(), ref, **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (5, 100, 37), (70, 130, 259), (128, 512, 1024)])
def test_linear(ops, dtype, M, N, K):
    x = torch.randn(M, K, device="cuda").to(dtype)
    w = (torch.randn(N, K, device="cuda") / math.sqrt(K)).to(dtype)
    res = torch.randn(M, N, device="cuda").to(dtype)
    ref = x.double().cpu() @ w.double().cpu().T
    t = dict(atol=1e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=3e-2, rtol=2e-2)
    assert torch.allclose(ops.linear(x, w).double().cpu(), ref, **t)
    assert torch.allclose(ops.linear(x, w, res).double().cpu(), ref + res.double().cpu(), **t)
    full = ops.linear(x, w, out_dtype=torch.float32)
    assert full.dtype == torch.float32
    assert torch.allclose(full.double().cpu(), ref, atol=1e-3 if dtype == torch.bfloat16 else 1e-5, rtol=1e-3)


def test_linear_rows_do_not_depend_on_the_batch(ops):
    """float32: a row's result is bit-equal whether it runs alone or among others."""
    x = torch.randn(70, 259, device="cuda")
    w = torch.randn(130, 259, device="cuda")
    whole = ops.linear(x, w)
    assert torch.equal(ops.linear(x[17:18].contiguous(), w), whole[17:18])
    assert torch.equal(ops.linear(x[60:].contiguous(), w), whole[60:])


@pytest.mark.parametrize("K", [1, 12, 30, 256, 260, 771, 772, 1028, 8192, 8460, 12288])
@pytest.mark.parametrize("N", [1, 63, 130, 384, 1600, 4800])
def test_float32_linear_in_both_kernels(ops, N, K):
    """The float32 product on either side of each of its dispatch's lines (4, 8, 16 and 32 rows; K by a multiple of 4,
    by fewer runs of 256 than quarters, by more than eight runs a block; rows off 16 bytes; matrices whose tiles of 32 rows
    are fewer than the SMs with some of these numbers of rows and more with others): against float64, within the
    bound of a sum cut into chains of 256, and each row the same bits whatever the number of rows beside it."""
    g = torch.Generator().manual_seed(N + K)
    if N > 384 and K > 1028:
        K = 4096 + K % 7  # (as many blocks, fewer multiply-adds for the float64 product)
    x = torch.randn(131, K, generator=g).cuda()
    w = torch.randn(N, K, generator=g).cuda()
    res = torch.randn(131, N, generator=g).cuda()
    exact = x.double() @ w.double().T
    runs = -(-K // 256)
    # a rounding per multiply-add of a chain, per run of a quarter, per quarter and for the residual
    bound = (256 + -(-runs // 4) + 4 + 1) * 2.0**-24 * (x.double().abs() @ w.double().abs().T + res.double().abs())
    whole, with_res = ops.linear(x, w), ops.linear(x, w, res)
    assert ((whole.double() - exact).abs() <= bound).all()
    assert ((with_res.double() - (exact + res.double())).abs() <= bound).all()
    for M in (1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65):
        assert torch.equal(ops.linear(x[:M], w), whole[:M]), M
        assert torch.equal(ops.linear(x[130 - M : 130], w, res[130 - M : 130]), with_res[130 - M : 130]), M
    off = torch.empty(131 * K + 1, device="cuda")[1:].view(131, K).copy_(x)  # rows that start off 16 bytes
    for M in (3, 20, 131):
        assert torch.equal(ops.linear(off[:M], w), whole[:M])


@pytest.mark.parametrize("M", [3, 8, 13, 30, 70, 131])
@pytest.mark.parametrize("N,K", [(130, 772), (63, 771), (384, 8460), (5, 96)])
def test_float32_linear_keeps_what_is_not_finite_in_its_row_and_column(ops, M, N, K):
    """A NaN among the inputs of one row, an infinity in one row of the matrix: that row, that column, and no other."""
    g = torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    plain_out = ops.linear(x, w)
    x[M // 2, K - 1], w[N // 2, K // 3] = math.nan, math.inf
    bad = torch.zeros(M, N, dtype=torch.bool, device="cuda")
    bad[M // 2], bad[:, N // 2] = True, True
    out = ops.linear(x, w)
    assert torch.equal(~torch.isfinite(out), bad) and torch.equal(out[~bad], plain_out[~bad])


@pytest.mark.parametrize("M", [1, 4, 7, 16, 17])
def test_float32_linear_waits_for_the_matrix_that_the_previous_kernel_writes(ops, M):
    """A matrix that comes from the library kernel right before (which lets its successor start early) is read when that
    kernel has completed, with as few rows as well."""
    g = torch.Generator().manual_seed(M)
    x, b = torch.randn(M, 2048, generator=g).cuda(), torch.randn(2048, 1024, generator=g).cuda()
    for i in range(6):
        a = torch.randn(512, 1024, generator=g).cuda()
        ref = ops.linear(x, ops.linear(a, b).clone())
        torch.cuda.synchronize()
        assert torch.equal(ops.linear(x, ops.linear(a, b)), ref), i


def rope_reference(x, positions, hd, theta, rotary_dim=None):
    rd = rotary_dim or hd
    angles = plain.rope_angles(positions, rd, theta)
    rotated = plain.apply_rope(x[..., :rd], angles)
    return torch.cat([rotated, x[..., rd:]], dim=-1)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hd,rd,theta", [(16, 16, 1e4), (48, 48, 5e4), (128, 128, 1e6), (256, 64, 1e4), (32, 32, 1e4),
                                         (64, 64, 1e6), (256, 256, 5e5)])  # fmt: skip
def test_rotary_alone(ops, dtype, hd, rd, theta):
    from atomserve_b200.parts.rotary import Rotary

    rot = Rotary(hidden_size=0, prefix="", head_dim=hd, theta=theta, rotary_dim=rd)
    rot.prepare(torch.device("cuda"))
    pos = torch.tensor([0, 1, 300, 4097, 39999], dtype=torch.int32, device="cuda")
    x = torch.randn(5, 3, hd, device="cuda").to(dtype)
    ref = rope_reference(x.float().cpu(), pos.cpu().long(), hd, theta, rd)
    out = rot.apply(x, pos)
    assert torch.allclose(out.float().cpu(), ref, **(dict(atol=2e-4, rtol=1e-4) if dtype == torch.float32 else tol(dtype)))
    assert torch.equal(out[0], x[0])  # position 0 is the identity


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,KV,hd,bs", [(4, 2, 16, 16), (5, 1, 48, 8), (32, 8, 128, 16), (16, 16, 80, 4), (6, 3, 32, 8),
                                        (9, 3, 64, 16), (4, 4, 256, 8)])  # fmt: skip
def test_qk_norm_rope_store(ops, dtype, H, KV, hd, bs):
    T, nblocks, eps, theta = 6, 9, 1e-5, 1e6
    qkv = torch.randn(T, (H + 2 * KV) * hd, device="cuda").to(dtype)
    qg, kg = (1 + 0.1 * torch.randn(hd, device="cuda") for _ in range(2))
    inv_freq = plain.rope_inv_freq(hd, theta).cuda()
    pos = torch.tensor([0, 1, 300, 4097, 39999, 17], dtype=torch.int32, device="cuda")
    slot_list = [bs * 7 + 1, 0, bs * 3 + bs - 1, 5 % bs + bs * 2, bs * 8, -1]
    slots = torch.tensor(slot_list, dtype=torch.int32, device="cuda")
    kc = torch.zeros(nblocks, KV, bs, hd, device="cuda", dtype=dtype)
    vc = torch.zeros_like(kc)
    q = ops.qk_norm_rope_store(qkv, H, KV, hd, pos, q_gain=qg, k_gain=kg, eps=eps, inv_freq=inv_freq,
                               rotary_dim=hd, slots=slots, k_cache=kc, v_cache=vc)  # fmt: skip
    x = qkv.float().cpu().view(T, H + 2 * KV, hd)
    angles = plain.rope_angles(pos.cpu().long(), hd, theta)
    q_ref = plain.apply_rope(plain.rms_norm(x[:, :H], qg.cpu(), eps), angles)
    k_ref = plain.apply_rope(plain.rms_norm(x[:, H : H + KV], kg.cpu(), eps), angles)
    t = dict(atol=3e-4, rtol=1e-4) if dtype == torch.float32 else tol(dtype)
    assert torch.allclose(q.float().cpu(), q_ref, **t)
    kflat = kc.float().cpu().permute(0, 2, 1, 3).reshape(nblocks * bs, KV, hd)
    vflat = vc.cpu().permute(0, 2, 1, 3).reshape(nblocks * bs, KV, hd)
    written = [s for s in slot_list if s >= 0]
    for i, s in enumerate(slot_list):
        if s >= 0:
            assert torch.allclose(kflat[s], k_ref[i], **t)
            assert torch.equal(vflat[s], qkv.cpu().view(T, H + 2 * KV, hd)[i, H + KV :])  # v bit-equal
    untouched = torch.ones(nblocks * bs, dtype=torch.bool)
    untouched[written] = False
    assert float(kflat[untouched].abs().max()) == 0 and float(vflat[untouched].float().abs().max()) == 0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,KV,hd,bs,gains", [(32, 8, 128, 16, True), (5, 1, 64, 8, True), (3, 3, 256, 4, False),
                                              (6, 2, 32, 16, True), (7, 1, 48, 8, True)])  # fmt: skip
def test_qk_norm_rope_store_many_tokens(ops, dtype, H, KV, hd, bs, gains):
    """The forms that portions of hundreds of tokens take (a block per token, several heads a
    warp), at head counts that leave warps half used, with some tokens not stored."""
    T, eps, theta = 300, 1e-6, 5e5
    g = torch.Generator().manual_seed(hd + H)
    qkv = torch.randn(T, (H + 2 * KV) * hd, generator=g).cuda().to(dtype)
    qg, kg = ((1 + 0.1 * torch.randn(hd, generator=g)).cuda() if gains else None for _ in range(2))
    inv_freq = plain.rope_inv_freq(hd, theta).cuda()
    pos = torch.randint(0, 30000, (T,), generator=g).int().cuda()
    nblocks = T // bs + 3
    slot_list = torch.randperm(nblocks * bs, generator=g)[:T].tolist()
    for i in range(0, T, 7):
        slot_list[i] = -1
    slots = torch.tensor(slot_list, dtype=torch.int32, device="cuda")
    kc = torch.zeros(nblocks, KV, bs, hd, device="cuda", dtype=dtype)
    vc = torch.zeros_like(kc)
    q = ops.qk_norm_rope_store(qkv, H, KV, hd, pos, q_gain=qg, k_gain=kg, eps=eps if gains else 0.0, inv_freq=inv_freq,
                               rotary_dim=hd, slots=slots, k_cache=kc, v_cache=vc)  # fmt: skip
    x = qkv.float().cpu().view(T, H + 2 * KV, hd)
    angles = plain.rope_angles(pos.cpu().long(), hd, theta)
    normed = (lambda v, gain: plain.rms_norm(v, gain.cpu(), eps)) if gains else (lambda v, gain: v)
    q_ref = plain.apply_rope(normed(x[:, :H], qg), angles)
    k_ref = plain.apply_rope(normed(x[:, H : H + KV], kg), angles)
    t = dict(atol=3e-4, rtol=1e-4) if dtype == torch.float32 else tol(dtype)
    assert torch.allclose(q.float().cpu(), q_ref, **t)
    kflat = kc.float().cpu().permute(0, 2, 1, 3).reshape(nblocks * bs, KV, hd)
    vflat = vc.cpu().permute(0, 2, 1, 3).reshape(nblocks * bs, KV, hd)
    stored = torch.tensor([s >= 0 for s in slot_list])
    at = torch.tensor([s for s in slot_list if s >= 0])
    assert torch.allclose(kflat[at], k_ref[stored], **t)
    assert torch.equal(vflat[at], qkv.cpu().view(T, H + 2 * KV, hd)[stored][:, H + KV :])
    untouched = torch.ones(nblocks * bs, dtype=torch.bool)
    untouched[at] = False
    assert float(kflat[untouched].abs().max()) == 0 and float(vflat[untouched].float().abs().max()) == 0


def paged_setup(ctx_lens, q_lens, H, KV, hd, bs, dtype, seed=0, special=None):
    """Random q/k/v for R requests; keys/values scattered over shuffled pages. Returns device
    inputs and the dense per-request k, v for the reference. `special` = (request, position):
    that key and the request's last query are made to match strongly."""
    g = torch.Generator().manual_seed(seed)
    R = len(ctx_lens)
    nblocks = sum(-(-c // bs) for c in ctx_lens) + 3
    order = torch.randperm(nblocks, generator=g).tolist()
    kc = torch.zeros(nblocks, KV, bs, hd)
    vc = torch.zeros(nblocks, KV, bs, hd)
    width = max(-(-c // bs) for c in ctx_lens)
    tables = torch.zeros(R, width, dtype=torch.int32)
    dense, qs = [], []
    for r, (c, n) in enumerate(zip(ctx_lens, q_lens)):
        k = torch.randn(c, KV, hd, generator=g)
        v = torch.randn(c, KV, hd, generator=g)
        q = torch.randn(n, H, hd, generator=g)
        if special is not None and special[0] == r:
            u = torch.randn(hd, generator=g)
            u = u / u.norm() * math.sqrt(hd) * 4
            k[special[1]] = u
            q[-1] = u
        k, v, q = (t.to(dtype).float() for t in (k, v, q))
        blocks = [order.pop() for _ in range(-(-c // bs))]
        tables[r, : len(blocks)] = torch.tensor(blocks, dtype=torch.int32)
        for p in range(c):
            kc[blocks[p // bs], :, p % bs] = k[p]
            vc[blocks[p // bs], :, p % bs] = v[p]
        dense.append((k, v))
        qs.append(q)
    q_start = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    pos_start = torch.tensor([c - n for c, n in zip(ctx_lens, q_lens)], dtype=torch.int32)
    dev = dict(
        q=torch.cat(qs).to(dtype).cuda(), k_cache=kc.to(dtype).cuda(), v_cache=vc.to(dtype).cuda(),
        block_tables=tables.cuda(), req_q_start=q_start.cuda(), req_pos_start=pos_start.cuda(),
    )  # fmt: skip
    return dev, dense, qs


def attention_reference(qs, dense, ctx_lens, q_lens, window):
    outs = []
    for q, (k, v), c, n in zip(qs, dense, ctx_lens, q_lens):
        # run the whole context as queries with zeros in front, keep the last n rows
        full_q = torch.cat([torch.zeros(c - n, *q.shape[1:]), q])
        outs.append(plain.attention(full_q, k, v, window)[c - n :])
    return torch.cat(outs)


ATTN_CASES = [
    # H, KV, hd, bs, ctx_lens, q_lens, window
    (4, 2, 16, 16, [1, 37, 512, 513, 1500], [1, 1, 1, 1, 1], None),
    (32, 8, 128, 16, [700, 33], [1, 33], None),
    (5, 1, 48, 8, [64, 130, 9], [64, 2, 9], None),
    (8, 8, 80, 4, [300, 45], [7, 45], None),
    (6, 3, 32, 8, [200, 77, 24, 25], [1, 30, 24, 2], 24),
    (64, 1, 64, 32, [129], [3], None),
    (16, 8, 256, 16, [90], [90], 17),
    # head sizes 64 and 128: the tensor-core kernels in bfloat16
    (10, 2, 64, 8, [300, 77, 150, 9], [1, 40, 5, 9], None),
    (64, 1, 64, 32, [129, 500], [3, 100], None),
    (32, 8, 128, 16, [2065, 1000, 65], [1, 1, 1], None),
    (16, 4, 128, 16, [600, 200], [600, 8], 100),
    (6, 3, 64, 4, [200, 77, 24, 25], [1, 30, 24, 2], 24),
    (8, 8, 128, 16, [130], [130], None),
    # prompt portions beside single tokens of long requests: the single tokens keep their key partitions
    (8, 2, 128, 16, [2065, 1000, 300, 3000], [1, 1, 200, 1], None),
    (8, 2, 128, 16, [3000, 64, 2500], [1, 64, 3], 700),
    # short rows before, between and after portions, five heads a group: the decode kernel's blocks count short rows only
    (40, 8, 128, 16, [900, 1200, 64, 700, 2100], [2, 300, 1, 8, 1], None),
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ATTN_CASES)
def test_paged_attention(ops, dtype, case):
    H, KV, hd, bs, ctx_lens, q_lens, window = case
    dev, dense, qs = paged_setup(ctx_lens, q_lens, H, KV, hd, bs, dtype)
    ref = attention_reference(qs, dense, ctx_lens, q_lens, window)
    common = dict(num_requests=len(ctx_lens), max_context=max(ctx_lens), window=window, scale=hd**-0.5)
    t = dict(atol=2e-5, rtol=1e-4) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)
    parts = (64, (max(ctx_lens) - 1) // 64 + 1)  # the keys split into partitions of 64 and merged
    for generic in (True, False):  # the general kernel, then whichever kernel serving would pick
        out = ops.paged_attention(**dev, **common, generic=generic, host_q_lens=q_lens)
        assert torch.allclose(out.float().cpu(), ref, **t), f"generic={generic}"
        if generic or max(q_lens) <= 8 or (dtype == torch.bfloat16 and hd == 128 and min(q_lens) <= 8):
            out2 = ops.paged_attention(**dev, **common, generic=generic, host_q_lens=q_lens, partitions=parts)
            assert torch.allclose(out2.float().cpu(), ref, **t), f"generic={generic} partitioned"
    out3 = ops.paged_attention(**dev, **common)  # without host knowledge of the portions
    assert torch.allclose(out3.float().cpu(), ref, **t)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("where", [0, 15, 16, 17, 255, 256, 511, 640, 999])
def test_attention_finds_one_far_key(ops, dtype, where):
    """One key among a thousand matches the query strongly: the output must be its value,
    wherever in its page and partition it lies."""
    H, KV, hd, bs, ctx = 8, 2, 64, 16, 1000
    dev, dense, qs = paged_setup([ctx], [1], H, KV, hd, bs, dtype, seed=where, special=(0, where))
    for parts, generic in ((None, False), ((256, 4), False), (None, True), ((256, 4), True)):
        out = ops.paged_attention(**dev, num_requests=1, max_context=ctx, window=None, scale=hd**-0.5,
                                  partitions=parts, generic=generic, host_q_lens=[1])  # fmt: skip
        v = dense[0][1][where]  # [KV, hd]
        expect = v.repeat_interleave(H // KV, dim=0)
        assert torch.allclose(out[0].float().cpu(), expect, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_window_edge(ops, dtype):
    """The key at p - window + 1 is seen, the key at p - window is not."""
    for hd in (32, 64):
        H, KV, bs, ctx, window = 4, 2, 8, 120, 24
        p = ctx - 1
        for where, seen in ((p - window + 1, True), (p - window, False)):
            for n in (1, 12):  # as a single decoded token, and as the last row of a portion
                dev, dense, qs = paged_setup([ctx], [n], H, KV, hd, bs, dtype, seed=3, special=(0, where))
                out = ops.paged_attention(**dev, num_requests=1, max_context=ctx, window=window, scale=hd**-0.5,
                                          host_q_lens=[n])  # fmt: skip
                expect = dense[0][1][where].repeat_interleave(H // KV, dim=0)
                close = torch.allclose(out[-1].float().cpu(), expect, atol=2e-2, rtol=2e-2)
                assert close == seen, (hd, where, n)


@pytest.mark.parametrize("prefill_kernel", ["tcgen05", "mma"])
@pytest.mark.parametrize("window", [100, 108])
def test_attention_window_edge_head_128(ops, monkeypatch, prefill_kernel, window):
    """The served head size, through the tensor-core kernels: a single decoded token (the mma
    decode kernel), the last row of a short portion and of a 200-token portion (the tcgen05
    kernel, then the mma prefill kernel). With 300 keys the window of 100 begins at key 200, inside
    a 64-key tile and inside a page; the window of 108 begins at key 192, the first key of a tile
    and of a page, so the unseen key is the last of the tile and page before."""
    import atomserve_b200.ops.attention as A

    monkeypatch.setattr(A, "PREFILL_KERNEL", prefill_kernel)
    H, KV, hd, bs, ctx = 8, 2, 128, 16, 300
    p = ctx - 1
    for where, seen in ((p - window + 1, True), (p - window, False)):
        for n in (1, 12, 200):
            dev, dense, qs = paged_setup([ctx], [n], H, KV, hd, bs, torch.bfloat16, seed=5, special=(0, where))
            out = ops.paged_attention(**dev, num_requests=1, max_context=ctx, window=window, scale=hd**-0.5,
                                      host_q_lens=[n])  # fmt: skip
            expect = dense[0][1][where].repeat_interleave(H // KV, dim=0)
            close = torch.allclose(out[-1].float().cpu(), expect, atol=2e-2, rtol=2e-2)
            assert close == seen, (prefill_kernel, window, where, n)
            ref = attention_reference(qs, dense, [ctx], [n], window)  # and every other row of the portion
            assert torch.allclose(out.float().cpu(), ref, atol=2e-2, rtol=2e-2), (prefill_kernel, window, where, n)
    from atomserve_b200.ops.linear import check_gemm_status

    check_gemm_status()


def long_context_setup(ctx_lens, q_lens, H, KV, hd, bs, seed, special=None):
    """Long requests without per-position Python loops: one pool of random pages on the device,
    shared by all requests, each request reading it through a shuffled block table of its own (so
    every request sees other keys in another order). Returns the device inputs and, per request,
    its keys and values in position order as float32 on the CPU. `special` = (request, position):
    that key matches the request's last query strongly."""
    g = torch.Generator().manual_seed(seed)
    pages = max(-(-c // bs) for c in ctx_lens)
    pool = pages + 5
    kc = (torch.randn(pool, KV, bs, hd, generator=g) * 0.5).bfloat16()
    vc = torch.randn(pool, KV, bs, hd, generator=g).bfloat16()
    tables = torch.stack([torch.randperm(pool, generator=g)[:pages] for _ in ctx_lens]).to(torch.int32)
    q = torch.randn(sum(q_lens), H, hd, generator=g).bfloat16()
    q_start = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    if special is not None:
        r, where = special
        u = torch.randn(hd, generator=g)
        u = (u / u.norm() * math.sqrt(hd) * 4).bfloat16()
        kc[tables[r, where // bs], :, where % bs] = u
        q[int(q_start[r + 1]) - 1] = u
    dense = []
    for r, c in enumerate(ctx_lens):
        mine = tables[r].long()
        k = kc[mine].permute(0, 2, 1, 3).reshape(-1, KV, hd)[:c].float()
        v = vc[mine].permute(0, 2, 1, 3).reshape(-1, KV, hd)[:c].float()
        dense.append((k, v))
    pos_start = torch.tensor([c - n for c, n in zip(ctx_lens, q_lens)], dtype=torch.int32)
    dev = dict(q=q.cuda(), k_cache=kc.cuda(), v_cache=vc.cuda(), block_tables=tables.cuda(),
               req_q_start=q_start.cuda(), req_pos_start=pos_start.cuda())  # fmt: skip
    return dev, dense, q.float()


def long_context_reference(q, dense, ctx_lens, q_lens, window=None):
    outs, at = [], 0
    for (k, v), c, n in zip(dense, ctx_lens, q_lens):
        outs.append(plain.attention_rows(q[at : at + n], k, v, torch.arange(c - n, c), window))
        at += n
    return torch.cat(outs)


@pytest.mark.parametrize("context", [8192, 32768])
@pytest.mark.parametrize("batch", [1, 8, 64])
def test_decode_attention_at_long_contexts(ops, batch, context):
    """Single decoded tokens over 8k and 32k keys with the ranges that the planner picks
    for 1, 8 and 64 requests, against the plain attention; the requests' contexts differ, the
    longest being `context`, and in request 0 one far key carries nearly all the weight."""
    from atomserve_b200.ops.attention import plan_decode_ranges

    H, KV, hd, bs = 8, 2, 128, 16
    ctx_lens = [context - (37 * r) % (context // 2) for r in range(batch)]
    where = context // 3 + 5
    dev, dense, q = long_context_setup(ctx_lens, [1] * batch, H, KV, hd, bs, seed=batch, special=(0, where))
    assert plan_decode_ranges(batch, KV, H // KV, context, 0, hd) > 1  # some row is cut, and merged
    out = ops.paged_attention(**dev, num_requests=batch, max_context=context, window=None, scale=hd**-0.5,
                              host_q_lens=[1] * batch).float().cpu()  # fmt: skip
    ref = long_context_reference(q, dense, ctx_lens, [1] * batch)
    assert torch.allclose(out, ref, atol=2e-2, rtol=2e-2), float((out - ref).abs().max())
    expect = dense[0][1][where].repeat_interleave(H // KV, dim=0)
    assert torch.allclose(out[0], expect, atol=2e-2, rtol=2e-2)
    general = ops.paged_attention(**dev, num_requests=batch, max_context=context, window=None, scale=hd**-0.5,
                                  host_q_lens=[1] * batch, generic=True).float().cpu()  # fmt: skip
    assert torch.allclose(general, ref, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("prefill_kernel", ["tcgen05", "mma"])
@pytest.mark.parametrize("ctx,n", [(8192, 8192), (8192, 512)])
def test_prefill_attention_at_long_contexts(ops, monkeypatch, prefill_kernel, ctx, n):
    """One prompt of 8,192 tokens in one step, and a portion of 512 tokens behind 7,680 cached
    ones, against the plain attention row by row."""
    import atomserve_b200.ops.attention as A
    from atomserve_b200.ops.linear import check_gemm_status

    monkeypatch.setattr(A, "PREFILL_KERNEL", prefill_kernel)
    H, KV, hd, bs = 4, 1, 128, 16
    dev, dense, q = long_context_setup([ctx], [n], H, KV, hd, bs, seed=n, special=(0, 100))
    out = ops.paged_attention(**dev, num_requests=1, max_context=ctx, window=None, scale=hd**-0.5,
                              host_q_lens=[n]).float().cpu()  # fmt: skip
    check_gemm_status()
    ref = long_context_reference(q, dense, [ctx], [n])
    assert torch.allclose(out, ref, atol=2e-2, rtol=2e-2), float((out - ref).abs().max())
    assert torch.allclose(out[-1], dense[0][1][100].repeat_interleave(H // KV, dim=0), atol=2e-2, rtol=2e-2)


def test_sampling_greedy_and_support(ops):
    logits = torch.tensor([[0.1, 3.0, 0.2, 3.0], [5.0, 1.0, 0.0, -1.0]], device="cuda")
    assert ops.argmax_rows(logits).tolist() == [1, 0]  # lowest id among equals

    probs = torch.tensor([0.4, 0.3, 0.2, 0.1])

    def draws(n, temperature, top_k, top_p, seed=1):
        lg = probs.log().repeat(n, 1).cuda().contiguous()
        return ops.sample_rows(
            lg, torch.full((n,), temperature, device="cuda"), torch.full((n,), top_k, dtype=torch.int32, device="cuda"),
            torch.full((n,), top_p, device="cuda"), torch.full((n,), seed, dtype=torch.int64, device="cuda"),
            torch.arange(n, dtype=torch.int64, device="cuda"),
        ).cpu()  # fmt: skip

    counts = draws(20000, 1.0, 0, 1.0).bincount(minlength=4)
    assert torch.allclose(counts / 20000, probs, atol=0.015)
    assert set(draws(2000, 1.0, 2, 1.0).tolist()) == {0, 1}
    assert set(draws(200, 1.0, 1, 1.0).tolist()) == {0}
    assert set(draws(2000, 1.0, 0, 0.6).tolist()) == {0, 1}
    assert set(draws(200, 1.0, 0, 0.01).tolist()) == {0}
    assert set(draws(50, 0.0, 3, 0.5).tolist()) == {0}
    # temperature reshapes the distribution: p^(1/T) renormalised
    counts = draws(20000, 0.5, 0, 1.0).bincount(minlength=4)
    sharp = probs**2 / (probs**2).sum()
    assert torch.allclose(counts / 20000, sharp, atol=0.015)


@pytest.mark.parametrize("V,k,p,temp", [(331, 20, 0.95, 0.6), (5000, 64, 0.8, 0.7), (151936, 20, 0.95, 0.6),
                                        (2000, 0, 0.9, 1.0), (3000, 1500, 0.5, 1.3)])  # fmt: skip
def test_sampling_support_matches_plain(ops, V, k, p, temp):
    """Everything drawn lies in the plain sampler's support, and frequent tokens agree."""
    g = torch.Generator().manual_seed(V)
    logits = torch.randn(V, generator=g) * 3
    dist = plain.sampling_distribution(logits, temp, k, p)
    n = 4000
    out = ops.sample_rows(
        logits.repeat(n, 1).cuda().contiguous(), torch.full((n,), temp, device="cuda"),
        torch.full((n,), k, dtype=torch.int32, device="cuda"), torch.full((n,), p, device="cuda"),
        torch.full((n,), 9, dtype=torch.int64, device="cuda"), torch.arange(n, dtype=torch.int64, device="cuda"),
    ).cpu().long()  # fmt: skip
    assert bool((dist[out] > 0).all())
    freq = out.bincount(minlength=V) / n
    assert float((freq - dist).abs().max()) < 0.04


def test_sampling_ties_at_the_cut(ops):
    """Equal logits at the k-th place: exactly k tokens stay, the lower ids."""
    logits = torch.tensor([[1.0, 2.0, 2.0, 2.0, 2.0, 0.5, 3.0]], device="cuda").repeat(500, 1).contiguous()
    n = 500
    out = ops.sample_rows(
        logits, torch.ones(n, device="cuda"), torch.full((n,), 3, dtype=torch.int32, device="cuda"),
        torch.ones(n, device="cuda"), torch.zeros(n, dtype=torch.int64, device="cuda"),
        torch.arange(n, dtype=torch.int64, device="cuda"),
    ).cpu()  # fmt: skip
    assert set(out.tolist()) == {6, 1, 2}


def test_seeded_rows_do_not_depend_on_neighbours(ops):
    g = torch.Generator().manual_seed(0)
    row = torch.randn(1000, generator=g)
    others = torch.randn(2, 1000, generator=g)

    def run(rows, seeds, counters):
        n = rows.shape[0]
        return ops.sample_rows(
            rows.cuda().contiguous(), torch.ones(n, device="cuda"), torch.full((n,), 50, dtype=torch.int32, device="cuda"),
            torch.ones(n, device="cuda"), torch.tensor(seeds, dtype=torch.int64, device="cuda"),
            torch.tensor(counters, dtype=torch.int64, device="cuda"),
        ).tolist()  # fmt: skip

    alone = [run(row[None], [7], [i])[0] for i in range(20)]
    crowd = [run(torch.stack([others[0], row, others[1]]), [1, 7, 2], [i + 5, i, i + 9])[1] for i in range(20)]
    assert alone == crowd and len(set(alone)) > 3


def philox_uniforms(seed: int, counter: int, n: int) -> np.ndarray:
    """The race's uniforms of tokens 0..n-1: Philox-4x32-10 (Salmon et al. 2011), counter (token, draw counter, 0x5a17)."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.arange(n, dtype=np.uint64), np.full(n, counter & 0xFFFFFFFF, np.uint64), np.full(n, counter >> 32, np.uint64),
         np.full(n, 0x5A17, np.uint64)]  # fmt: skip
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return ((c[0] >> np.uint64(8)).astype(np.float64) + 0.5) / 2.0**24


@pytest.mark.parametrize("V", [1, 3, 30, 33, 257, 4099, 32000, 400004])
@pytest.mark.parametrize("k,p,temp", [(20, 0.95, 0.6), (0, 0.9, 1.0), (1024, 0.999, 1.0), (1025, 0.8, 1.3), (1, 1.0, 0.7), (0, 1.0, 1.0)])
def test_sampled_token_wins_the_plain_race(ops, V, k, p, temp):
    """The drawn token is the winner of the exponential race over the plain sampler's support, at row lengths around
    the edges of a block's share of a row (eighths, multiples of four) and beyond what shared memory holds, with ties
    and masked (-inf) tokens among the logits, and each way top-k can go."""
    g = torch.Generator().manual_seed(V + k)
    logits = torch.randn(3, V, generator=g) * 3
    logits[1] = (logits[1] * 2).round() / 2  # ties at every cut
    if V > 3:
        logits[2, torch.randperm(V, generator=g)[: V // 2]] = -math.inf
    seeds, counters = [5, (1 << 40) + 3, 77], [0, 9, 1 << 33]
    out = ops.sample_rows(
        logits.cuda(), torch.full((3,), temp, device="cuda"), torch.full((3,), k, dtype=torch.int32, device="cuda"),
        torch.full((3,), p, device="cuda"), torch.tensor(seeds, device="cuda"), torch.tensor(counters, device="cuda"),
    ).tolist()  # fmt: skip
    assert ops.argmax_rows(logits.cuda()).tolist() == [int(torch.nonzero(r == r.max())[0]) for r in logits]
    for r in range(3):
        x = logits[r].double().numpy()
        order = np.lexsort((np.arange(V), -x))  # largest first, lower ids first among equals
        order = order[: k if 0 < k < V else V]
        mass = np.exp((x[order] - x[order[0]]) / np.float64(np.float32(temp)))
        before = np.cumsum(mass) - mass
        kept = order[before < p * mass.sum() * (1 - 1e-9)] if p < 1 else order
        edge = order[before < p * mass.sum() * (1 + 1e-6)] if p < 1 else order  # float32 masses may keep one more at the cut
        score = np.exp((x - x.max()) / np.float64(np.float32(temp))) / np.maximum(-np.log(philox_uniforms(seeds[r], counters[r], V)), 1e-10)
        assert out[r] in edge
        # (the kernel's float32 exponential and logarithm differ from these by a few units in the last place)
        assert score[out[r]] >= score[kept].max() * (1 - 1e-5)


@pytest.mark.parametrize("V", [2, 1024, 1025, 4099, 32000])
@pytest.mark.parametrize("spread,k,p,temp", [(0.0, 0, 0.5, 1.0), (1e-6, 0, 0.9, 0.8), (1e-3, 1500, 0.3, 1.0), (3.0, 0, 0.5, 50.0),
                                             (3.0, 0, 0.99, 0.02), (30.0, 0, 0.9, 1.0)])  # fmt: skip
def test_the_cut_of_top_p_wherever_the_mass_lies(ops, V, spread, k, p, temp):
    """The steps below the largest logit in which the walk over masses begins: all logits in one step (as many as the buffer
    of candidates holds, and one more), steps of a few neighbouring floats, nearly all mass in the first or far down."""
    g = torch.Generator().manual_seed(V + k)
    logits = (torch.randn(2, V, generator=g) * spread + 7).float()
    seeds, counters = [5, (1 << 40) + 3], [0, 9]
    out = ops.sample_rows(
        logits.cuda(), torch.full((2,), temp, device="cuda"), torch.full((2,), k, dtype=torch.int32, device="cuda"),
        torch.full((2,), p, device="cuda"), torch.tensor(seeds, device="cuda"), torch.tensor(counters, device="cuda"),
    ).tolist()  # fmt: skip
    for r in range(2):
        x = logits[r].double().numpy()
        order = np.lexsort((np.arange(V), -x))[: k if 0 < k < V else V]
        mass = np.exp((x[order] - x[order[0]]) / np.float64(np.float32(temp)))
        before, p32 = np.cumsum(mass) - mass, np.float64(np.float32(p))
        # float32 masses (a few units of 2^-24 each) may keep one token more or fewer at the cut
        kept, edge = order[before < p32 * mass.sum() * (1 - 1e-6)], order[before < p32 * mass.sum() * (1 + 1e-6)]
        score = np.exp((x - x.max()) / np.float64(np.float32(temp))) / np.maximum(-np.log(philox_uniforms(seeds[r], counters[r], V)), 1e-10)
        assert out[r] in edge
        assert score[out[r]] >= score[kept].max() * (1 - 1e-5)


@pytest.mark.parametrize("V", [5, 500, 4099, 50001, 151936])
@pytest.mark.parametrize("k,p,temp", [(20, 0.95, 0.6), (0, 0.95, 0.8), (2000, 0.9, 1.0), (0, 1.0, 1.0), (3, 1.0, 1.0), (0, 1.0, 0.0)])
def test_a_rows_token_does_not_depend_on_how_many_rows_there_are(ops, V, k, p, temp):
    """How many blocks share a row goes by the number of rows: the same row, seed and counter draw the same token in a
    batch of one and of hundreds, with masked tokens, infinities and NaN among the logits and with ties at every cut."""
    g = torch.Generator().manual_seed(V)
    rows = torch.randn(7, V, generator=g) * 3
    rows[1] = (rows[1] * 2).round() / 2
    rows[2, torch.randperm(V, generator=g)[: V // 2]] = -math.inf
    rows[3, V // 3] = math.nan
    rows[4, V // 2] = math.inf
    rows[5], rows[6] = -math.inf, math.nan

    def draw(logits, seeds):
        n = logits.shape[0]
        setting = lambda v, dt: torch.full((n,), v, dtype=dt, device="cuda")  # noqa: E731
        args = setting(temp, torch.float32), setting(k, torch.int32), setting(p, torch.float32), seeds, seeds * 3
        return ops.sample_rows(logits, *args).cpu(), ops.argmax_rows(logits).cpu()

    seeds = torch.arange(7, device="cuda") + 11
    alone = [draw(rows[r : r + 1].cuda(), seeds[r : r + 1]) for r in range(7)]
    sampled, best = (torch.cat(t) for t in zip(*alone))
    assert sampled[5] == sampled[6] == 0 and sampled[3] != V // 3  # nothing to choose from; a NaN is not chosen
    finite = [torch.where(torch.isnan(r), -math.inf, r) for r in rows]
    assert best.tolist() == [int(torch.nonzero(r == r.max())[0]) for r in finite]
    if p < 1:
        assert sampled[4] == V // 2
    for n in (30, 70, 140, 290, 600):
        which = torch.arange(n) % 7
        got = draw(rows[which].cuda(), seeds[which.cuda()])
        assert torch.equal(got[0], sampled[which]) and torch.equal(got[1], best[which]), n


def test_presence_penalty(ops):
    logits = torch.zeros(2, 10, device="cuda")
    ops.presence_penalty(
        logits, torch.tensor([0, 0, 1], dtype=torch.int32, device="cuda"),
        torch.tensor([3, 4, 9], dtype=torch.int32, device="cuda"), torch.tensor([1.5, 1.5, 0.5], device="cuda"),
    )  # fmt: skip
    expect = torch.zeros(2, 10)
    expect[0, 3] = expect[0, 4] = -1.5
    expect[1, 9] = -0.5
    assert torch.equal(logits.cpu(), expect)


GEMM_SHAPES = [
    (1, 128, 64), (3, 100, 72), (16, 256, 512), (17, 384, 4096), (33, 130, 1024), (64, 4096, 4096),
    (8, 4096, 12288), (65, 256, 128), (128, 300, 264), (300, 512, 1000), (2048, 1024, 512),
    (200, 4096, 1024), (256, 512, 2048), (100, 24576, 256), (40, 20000, 128),
    (300, 4096, 512), (512, 4104, 256), (700, 5120, 128), (384, 6144, 192),
    (300, 4096, 8192), (512, 1000, 8256), (257, 2048, 12288),
]  # fmt: skip


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
def test_gemm_tcgen05(ops, M, N, K):
    """The tcgen05/TMEM/TMA GEMM against float64, in every epilogue, swapped and split shapes
    included; its status word must stay zero (no pipeline wait ran out)."""
    from atomserve_b200.ops.linear import check_gemm_status, gemm_tcgen05

    g = torch.Generator().manual_seed(M * 7 + N + K)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).bfloat16().cuda()
    res = torch.randn(M, N, generator=g).bfloat16().cuda()
    ref = x.double().cpu() @ w.double().cpu().T
    full = gemm_tcgen05(x, w, None, torch.float32)
    check_gemm_status()
    assert torch.allclose(full.double().cpu(), ref, atol=2e-3, rtol=1e-3), float((full.double().cpu() - ref).abs().max())
    plain_out = gemm_tcgen05(x, w, None, torch.bfloat16)
    with_res = gemm_tcgen05(x, w, res, torch.bfloat16)
    check_gemm_status()
    assert torch.allclose(plain_out.double().cpu(), ref, atol=3e-2, rtol=2e-2)
    assert torch.allclose(with_res.double().cpu(), ref + res.double().cpu(), atol=3e-2, rtol=2e-2)
    # a row's result does not depend on the rows beside it (same kernel shape: same tile path)
    if M > 1:
        again = gemm_tcgen05(x, w, None, torch.float32)
        assert torch.equal(again, full)


TCGEN05_ATTN_CASES = [
    # H, KV, bs, ctx_lens, q_lens, window
    (4, 1, 16, [200], [200], None),
    (32, 8, 16, [700, 33, 2100], [1, 33, 300], None),
    (8, 8, 8, [130, 500], [130, 260], None),
    (16, 8, 32, [640, 129, 77], [129, 129, 9], None),
    (16, 2, 64, [1000], [333], 200),
    (16, 1, 128, [300, 150], [100, 150], 64),
    (8, 2, 16, [2048], [2048], None),
    # groups that do not divide 128: 25, 42 and 18 tokens a tile, the last rows of a tile padding
    (40, 8, 16, [700, 90, 300], [300, 90, 1], None),
    (6, 2, 16, [500], [500], 130),
    (7, 1, 32, [333, 64], [200, 64], None),
]


@pytest.mark.parametrize("case", TCGEN05_ATTN_CASES)
def test_prefill_attention_tcgen05(ops, case):
    """The tcgen05 prefill kernel (scores and output in tensor memory, V as an MN-major operand,
    pages fetched by TMA) against the plain attention, and against the mma.sync kernel it
    replaces; prompt portions with a cached prefix, several requests, windows, every group size
    and page size it serves."""
    from atomserve_b200.ops import attention as attn
    from atomserve_b200.ops.linear import check_gemm_status

    H, KV, bs, ctx_lens, q_lens, window = case
    hd = 128
    dev, dense, qs = paged_setup(ctx_lens, q_lens, H, KV, hd, bs, torch.bfloat16, seed=H + bs)
    ref = attention_reference(qs, dense, ctx_lens, q_lens, window)
    common = dict(num_requests=len(ctx_lens), max_context=max(ctx_lens), window=window, scale=hd**-0.5, host_q_lens=q_lens)
    assert attn.lib().asb_attention_tcgen05_supported(hd, H // KV, bs)
    results = {}
    for kernel in ("tcgen05", "mma"):
        attn.PREFILL_KERNEL = kernel
        try:
            results[kernel] = ops.paged_attention(**dev, **common).float().cpu()
        finally:
            attn.PREFILL_KERNEL = "tcgen05"
    check_gemm_status()
    assert torch.allclose(results["tcgen05"], ref, atol=2e-2, rtol=2e-2), float((results["tcgen05"] - ref).abs().max())
    assert torch.allclose(results["mma"], ref, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("M,I,K", [(1, 64, 64), (5, 200, 72), (16, 1024, 512), (40, 352, 256), (64, 12288, 4096),
                                   (100, 176, 80), (300, 704, 256), (2048, 512, 512),
                                   (130, 25600, 5120), (302, 17408, 5120), (281, 17410, 5128)])  # fmt: skip
def test_gemm_tcgen05_swiglu(ops, M, I, K):
    """silu(x gate^T) * (x up^T) from the GEMM's own epilogue (and, where K is cut, from the
    reduction of its partial sums) against float64."""
    from atomserve_b200.ops.linear import check_gemm_status

    g = torch.Generator().manual_seed(M + I + K)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    gate = (torch.randn(I, K, generator=g) / math.sqrt(K) * 2).bfloat16().cuda()
    up = (torch.randn(I, K, generator=g) / math.sqrt(K) * 2).bfloat16().cuda()
    w = ops.interleave_gate_up(gate, up)
    assert torch.equal(w[0::2], gate) and torch.equal(w[1::2], up)
    if not ops.swiglu_fusable(w):
        pytest.skip("the tensor-core GEMM is switched off (ATOMSERVE_B200_GEMM)")
    out = ops.linear_swiglu(x, w)
    check_gemm_status()
    gs, us = x.double().cpu() @ gate.double().cpu().T, x.double().cpu() @ up.double().cpu().T
    ref = gs / (1 + torch.exp(-gs)) * us
    assert out.shape == (M, I) and torch.allclose(out.double().cpu(), ref, atol=2e-2, rtol=2e-2)


def _skip_without_partial_sums():
    import importlib

    L = importlib.import_module("atomserve_b200.ops.linear")
    if not L.PARTIAL_SUMS or L.BACKEND != "tcgen05":
        pytest.skip("partial sums are switched off (ATOMSERVE_B200_PARTIAL_SUMS, ATOMSERVE_B200_GEMM)")


PARTIAL_NORM_SHAPES = [(1, 4096, 4096), (8, 4096, 12288), (5, 1024, 2048), (16, 640, 1024), (33, 2048, 4096),
                       (64, 4096, 4096), (7, 5120, 17408), (3, 264, 2048), (100, 4096, 4096), (128, 1024, 2048)]  # fmt: skip


@pytest.mark.parametrize("M,N,K", PARTIAL_NORM_SHAPES)
def test_partial_add_rms_norm_is_the_unfused_result(ops, M, N, K):
    """A product left as the GEMM's partial sums, added up with the residual and normalised in
    one kernel: the same bits as the GEMM with its own reduction followed by rms_norm, and close
    to float64."""
    from atomserve_b200.ops.linear import check_gemm_status

    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).bfloat16().cuda()
    res = torch.randn(M, N, generator=g).bfloat16().cuda()
    gain = (1 + 0.1 * torch.randn(N, generator=g)).cuda()
    _skip_without_partial_sums()
    product = ops.linear_partial(x, w)
    assert product is not None, "these shapes cut K: the partial-sum form must be available"
    assert (product.tokens, product.columns) == (M, N)
    total, normed = ops.partial_add_rms_norm(product, res, gain, 1e-6)
    plain_total = ops.linear(x, w, res)
    plain_normed = ops.rms_norm(plain_total, gain, 1e-6)
    check_gemm_status()
    assert torch.equal(total, plain_total) and torch.equal(normed, plain_normed)
    ref = x.double().cpu() @ w.double().cpu().T + res.double().cpu()
    assert torch.allclose(total.double().cpu(), ref, atol=3e-2, rtol=2e-2)
    # without a residual
    total0, normed0 = ops.partial_add_rms_norm(ops.linear_partial(x, w), None, gain, 1e-6)
    plain0 = ops.linear(x, w)
    assert torch.equal(total0, plain0) and torch.equal(normed0, ops.rms_norm(plain0, gain, 1e-6))


def test_linear_partial_declines_what_does_not_cut_k(ops):
    """Many tokens, float32 operands and tiny products have no partial-sum form: None, and the
    caller takes the plain product."""
    x = torch.randn(300, 512, device="cuda").bfloat16()
    w = torch.randn(1024, 512, device="cuda").bfloat16()
    assert ops.linear_partial(x, w) is None
    assert ops.linear_partial(x[:4].float(), w.float()) is None


# beyond 128 tokens the planner rarely swaps the operands and cuts K (which is when the product can
# be left as partial sums): the last shape's 150 tokens run with that form forced
QKV_PARTIAL_SHAPES = [(8, 2, 128, 2048), (32, 8, 128, 4096), (4, 2, 64, 1024), (6, 3, 32, 2048), (2, 1, 256, 1024), (8, 0, 128, 2048),
                      (4, 1, 128, 12288)]  # fmt: skip


@pytest.mark.parametrize("T,H,KV,hd,K", [(T, *shape) for shape in QKV_PARTIAL_SHAPES for T in (1, 6, 40, 128, 150)
                                         if T <= 128 or shape[3] >= 12288])  # fmt: skip
def test_qk_norm_rope_store_from_partial_sums(ops, T, H, KV, hd, K):
    """q/k norm, rotation and the cache write reading the qkv product from the GEMM's partial
    sums: the same bits as from the reduced product (KV = 0: queries only, nothing stored)."""
    from atomserve_b200.ops.linear import check_gemm_status, gemm_tune

    _skip_without_partial_sums()
    g = torch.Generator().manual_seed(H * 100 + hd + T)
    bs, nblocks = 16, 12
    x = torch.randn(T, K, generator=g).bfloat16().cuda()
    w = (torch.randn((H + 2 * KV) * hd, K, generator=g) / math.sqrt(K)).bfloat16().cuda()
    qg, kg = ((1 + 0.1 * torch.randn(hd, generator=g)).cuda() for _ in range(2))
    inv_freq = plain.rope_inv_freq(hd, 1e6).cuda()
    pos = torch.randint(0, 40000, (T,), generator=g).int().cuda()
    slot_list = torch.randperm(nblocks * bs, generator=g)[:T].tolist()
    if T > 1:
        slot_list[1] = -1
    slots = torch.tensor(slot_list, dtype=torch.int32, device="cuda")
    results = []
    for partial in (False, True):
        kc = torch.zeros(nblocks, max(KV, 1), bs, hd, device="cuda", dtype=torch.bfloat16)
        vc = torch.zeros_like(kc)
        if T > 128:
            gemm_tune(1)  # swapped operands: tiles of 128 weight rows by 256 tokens
        try:
            qkv = ops.linear_partial(x, w) if partial else ops.linear(x, w)
        finally:
            gemm_tune()
        assert qkv is not None
        store = dict(slots=slots, k_cache=kc, v_cache=vc) if KV else dict(slots=None, k_cache=None, v_cache=None)
        q = ops.qk_norm_rope_store(qkv, H, KV, hd, pos, q_gain=qg, k_gain=kg, eps=1e-6, inv_freq=inv_freq,
                                   rotary_dim=hd, **store)  # fmt: skip
        results.append((q, kc, vc))
    check_gemm_status()
    for a, b in zip(*results):
        assert torch.equal(a, b)
    assert float(results[1][0].float().abs().max()) > 0


def test_captured_gemm_survives_workspace_growth(ops):
    """A CUDA graph captured while the GEMM's partial-sum workspace was small keeps working after
    a larger call has replaced it: the outgrown buffer stays alive for the graphs that use it."""
    import importlib

    L = importlib.import_module("atomserve_b200.ops.linear")  # `ops.linear` itself is the function
    g = torch.Generator().manual_seed(5)
    x = torch.randn(8, 4096, generator=g).bfloat16().cuda()
    w = (torch.randn(4096, 4096, generator=g) / 64).bfloat16().cuda()
    expect = L.gemm_tcgen05(x, w, None, torch.bfloat16).clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = L.gemm_tcgen05(x, w, None, torch.bfloat16)
    before = L.gemm_workspace(x.device, 1)
    L.gemm_workspace(x.device, before.numel() + 1)  # a larger call comes along
    assert L.gemm_workspace(x.device, 1) is not before
    junk = [torch.full((before.numel(),), float("nan"), device="cuda") for _ in range(2)]  # would land in freed memory
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, expect)
    del junk
    L.check_gemm_status()


def test_a_wait_that_runs_out_reports_frees_tensor_memory_and_returns(ops):
    """The give-up path of the tcgen05 kernels, executed on purpose by a kernel that waits (a few
    thousand polls) on a barrier nothing arrives at: the status word names it, the block frees its
    tensor memory and ends, the context stays usable, and a GEMM that needs all of an SM's tensor
    memory runs right afterwards. The engine's step would fail with this report."""
    from atomserve_b200.ops.linear import check_gemm_status, gemm_tcgen05
    from atomserve_b200.ops.status import bounded_wait_selftest, status_for

    check_gemm_status()
    for _ in range(3):  # repeatedly: tensor memory that was not freed would run out or stall
        report = bounded_wait_selftest("cuda", polls=2048)
        assert report is not None and "self-test" in report and "gave up a bounded wait" in report
    assert status_for("cuda").problem() is None  # cleared by the read
    x = torch.randn(128, 512, device="cuda").bfloat16()
    w = torch.randn(384, 512, device="cuda").bfloat16()
    out = gemm_tcgen05(x, w, None, torch.float32)
    check_gemm_status()
    assert torch.allclose(out.double().cpu(), x.double().cpu() @ w.double().cpu().T, atol=2e-2, rtol=1e-3)


# the last three leave a last round of few tiles, which the kernel cuts along K (for one or both tile widths)
PAIR_SHAPES = [(300, 512, 256), (257, 1000, 520), (129, 130, 72), (2048, 4096, 4096), (700, 6144, 4160),
               (513, 24576, 1024), (1000, 256, 64), (3000, 384, 200), (640, 4104, 8),
               (1000, 5000, 4160), (300, 4000, 4160), (520, 1100, 2120)]  # fmt: skip


@pytest.mark.parametrize("rows", [128, 160, 224, 256])
@pytest.mark.parametrize("M,N,K", PAIR_SHAPES)
def test_gemm_tcgen05_on_pairs_of_sms(ops, M, N, K, rows):
    """The many-token form of the GEMM (tcgen05.mma.cta_group::2: two CTAs on a tile of 256 tokens
    by 128 to 256 weight rows), forced for shapes the planner would also give to single SMs: every
    epilogue against float64; tokens, weight rows and K that end inside a tile, an odd number of K
    blocks (the second K block of the last stage lies beyond K), one tile, many tiles per pair, a
    last round of tiles cut along K into pieces that a second kernel adds up."""
    from atomserve_b200.ops.linear import check_gemm_status, gemm_tcgen05, gemm_tune

    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).bfloat16().cuda()
    res = torch.randn(M, N, generator=g).bfloat16().cuda()
    ref = x.double().cpu() @ w.double().cpu().T
    gemm_tune(2, rows)
    try:
        full = gemm_tcgen05(x, w, None, torch.float32)
        plain_out = gemm_tcgen05(x, w, None, torch.bfloat16)
        with_res = gemm_tcgen05(x, w, res, torch.bfloat16)
        fused = gemm_tcgen05(x, w, None, torch.bfloat16, swiglu=True) if N % 2 == 0 else None
        again = gemm_tcgen05(x, w, None, torch.float32)
        gemm_tune(2, rows, cut_last_round=False)
        uncut = gemm_tcgen05(x, w, None, torch.float32)
    finally:
        gemm_tune()
    check_gemm_status()
    # cut or whole, the same products are added, in another order
    assert torch.allclose(uncut, full, atol=1e-4, rtol=1e-4)
    assert torch.allclose(full.double().cpu(), ref, atol=2e-3, rtol=1e-3), float((full.double().cpu() - ref).abs().max())
    assert torch.equal(again, full)
    assert torch.allclose(plain_out.double().cpu(), ref, atol=3e-2, rtol=2e-2)
    assert torch.allclose(with_res.double().cpu(), ref + res.double().cpu(), atol=3e-2, rtol=2e-2)
    if fused is not None:
        gate, up = ref[:, 0::2], ref[:, 1::2]
        assert torch.allclose(fused.double().cpu(), gate / (1 + torch.exp(-gate)) * up, atol=3e-2, rtol=3e-2)


def ranges_end_with_rows(tiles, ranges):
    """Whether the decode kernel cuts these rows (of so many 64-key tiles) one by one, each into equal ranges of its own,
    or all of them as one sequence whose ranges run from one row into the next (tiles_a_range in csrc/attention_mma.cu)."""
    least = -(-sum(tiles) // ranges)
    return len(tiles) <= 128 and any(sum(-(-t // c) for t in tiles) <= ranges for c in range(max(1, least), least + 3))


def tiles_of(lens, q_lens, window):
    """64-key tiles of each row of the requests that bring at most eight tokens."""
    at = [p for n, m in zip(lens, q_lens) if m <= 8 for p in range(n - m, n)]
    return [p // 64 - (max(0, p - window + 1) if window else 0) // 64 + 1 for p in at]


@pytest.mark.parametrize("lens,H,KV,hd,bs,window,ranges,by_row", [
    ([1], 8, 2, 128, 16, None, 7, True),                                # more ranges than tiles
    ([1, 64, 65, 129, 4000], 8, 2, 128, 16, None, 13, True),            # most ranges within one row
    ([1, 64, 65, 129, 4000], 8, 2, 128, 16, None, 3, False),            # a range over several rows, then two within one
    ([1 + (53 * i) % 700 for i in range(300)], 4, 2, 64, 8, None, 50, False),  # more rows than a round of the scan, rows of 1 to 11 tiles
    ([500, 3, 2000, 777], 40, 2, 128, 16, 300, 31, True),               # twenty heads a kv head: two chunks; a window
    ([500, 3, 2000, 777], 40, 2, 128, 16, 300, 3, False),               # the same, ranges across rows
    ([900] * 6, 16, 1, 64, 4, None, 64, True),                          # sixteen heads, two tiles a range
    ([900] * 6, 16, 1, 64, 4, None, 4, False),                          # sixteen heads, every range but the last ends inside a row
    ([900, 130, 64, 1500, 70, 333], 16, 1, 128, 16, None, 5, False),
    ([900, 130, 64, 1500, 70, 333], 9, 1, 128, 16, None, 4, False),     # nine heads
    ([40 + 97 * i % 600 for i in range(128)], 8, 8, 128, 16, None, 37, False),  # as many rows as threads, one head a kv head
])  # fmt: skip
@pytest.mark.parametrize("stored", [False, True])
def test_decode_attention_ranges(ops, monkeypatch, lens, H, KV, hd, bs, window, ranges, by_row, stored):
    """The decode kernel's equal ranges of all rows' key tiles, for numbers of ranges that the planner would not take,
    against the plain attention. bfloat16 values and probabilities: 2^-8 of values of size one, a few times over."""
    import atomserve_b200.ops.attention as attention

    rows = len(lens)
    assert ranges_end_with_rows(tiles_of(lens, [1] * rows, window), ranges) == by_row
    dev, dense, qs = paged_setup(lens, [1] * rows, H, KV, hd, bs, torch.bfloat16)
    ref = attention_reference(qs, dense, lens, [1] * rows, window)
    monkeypatch.setattr(attention, "plan_decode_ranges", lambda *a: ranges)
    out = ops.paged_attention(**dev, num_requests=rows, max_context=max(lens), window=window, scale=hd**-0.5,
                              host_q_lens=[1] * rows, earlier_keys_stored=stored)  # fmt: skip
    assert torch.allclose(out.float().cpu(), ref, atol=2e-2, rtol=2e-2), float((out.float().cpu() - ref).abs().max())


@pytest.mark.parametrize("lens,q_lens,ranges,by_row", [
    ([900, 1200, 64, 700, 2100, 33], [2, 300, 1, 8, 1, 1], 11, False),  # short rows of one to eight tokens around a portion
    ([900, 1200, 64, 700, 2100, 33], [2, 300, 1, 8, 1, 1], 40, True),
    ([70 + i for i in range(140)] + [400], [1] * 140 + [64], 29, False),  # more rows than a round of the scan, beside a portion
])  # fmt: skip
@pytest.mark.parametrize("H", [10, 40])
@pytest.mark.parametrize("known", [True, False])
def test_decode_attention_ranges_in_mixed_steps(ops, monkeypatch, lens, q_lens, ranges, by_row, H, known):
    """The same beside prompt portions, whose rows the decode kernel leaves alone, with and without host knowledge of
    what each request brings (without it all rows of the step are more than one round of the scan)."""
    import atomserve_b200.ops.attention as attention

    assert ranges_end_with_rows(tiles_of(lens, q_lens, None), ranges) == by_row
    dev, dense, qs = paged_setup(lens, q_lens, H, 2, 128, 16, torch.bfloat16)
    ref = attention_reference(qs, dense, lens, q_lens, None)
    monkeypatch.setattr(attention, "plan_decode_ranges", lambda *a: ranges)
    out = ops.paged_attention(**dev, num_requests=len(lens), max_context=max(lens), window=None, scale=128**-0.5,
                              host_q_lens=q_lens if known else None, earlier_keys_stored=True)  # fmt: skip
    assert torch.allclose(out.float().cpu(), ref, atol=2e-2, rtol=2e-2), float((out.float().cpu() - ref).abs().max())


@pytest.mark.parametrize("hd,group", [(64, 4), (128, 4), (128, 20)])
def test_decode_launch_without_rows_keeps_the_order_of_kernels(ops, monkeypatch, hd, group):
    """A step of long portions whose lengths the host does not tell: the decode kernel is launched and finds no row of
    its own. What follows on the stream still comes after the portions' kernel: here a product of its output."""
    import atomserve_b200.ops.attention as attention

    monkeypatch.setattr(attention, "MIXED_OVERLAP", False)  # both kernels on one stream
    KV, lens, q_lens = 2, [700, 1200, 64, 2000], [300, 500, 9, 1200]
    H = KV * group
    dev, dense, qs = paged_setup(lens, q_lens, H, KV, hd, 16, torch.bfloat16)
    w = (torch.randn(256, H * hd, generator=torch.Generator().manual_seed(1)) * 0.05).bfloat16().cuda()
    common = dict(num_requests=len(lens), max_context=max(lens), window=None, scale=hd**-0.5)
    known = ops.paged_attention(**dev, **common, host_q_lens=q_lens)
    ref = ops.paged_attention(**dev, **common)
    torch.cuda.synchronize()
    assert torch.allclose(ref.float(), known.float(), atol=2e-2, rtol=2e-2)  # (a portion's keys may be divided among blocks)
    expect = ops.linear(ref.view(-1, H * hd), w)
    assert attention.plan_decode_ranges(sum(q_lens), KV, group, max(lens), 0, hd, (64, 4)) > 0
    for partitions in (None, (64, 4)):
        torch.cuda.synchronize()
        for _ in range(20):
            out = ops.paged_attention(**dev, **common, partitions=partitions)
            got = ops.linear(out.view(-1, H * hd), w)
            assert torch.equal(out, ref) and torch.equal(got, expect)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("q_lens", [[1] * 48, [1, 3, 8, 1] * 12, [200, 64, 9] * 4, [1, 90] * 12])
def test_attention_reads_indexes_that_the_previous_kernel_writes(ops, monkeypatch, q_lens, hd):
    """Positions that come from the library kernel right before (an argmax over wide rows, which lets its successor start
    early): without `earlier_keys_stored` every attention kernel reads them only when that kernel has completed."""
    import atomserve_b200.ops.attention as attention

    monkeypatch.setattr(attention, "MIXED_OVERLAP", False)  # all kernels on one stream
    R, V, H, KV, bs = len(q_lens), 200000, 8, 2, 16
    width = V // bs // 8
    g = torch.Generator().manual_seed(hd + R)
    kc, vc = (torch.randn(64, KV, bs, hd, generator=g).bfloat16().cuda() for _ in range(2))
    tables = torch.randint(0, 64, (R, width), generator=g).int().cuda()
    q = torch.randn(sum(q_lens), H, hd, generator=g).bfloat16().cuda()
    starts = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32).cuda()
    common = dict(num_requests=R, max_context=3300, window=None, scale=hd**-0.5, host_q_lens=q_lens)
    for i in range(6):
        at = torch.randint(0, 3000, (R,), generator=g)
        marked = torch.zeros(R, V, device="cuda")
        marked[torch.arange(R, device="cuda"), at.cuda()] = 1.0
        ref = ops.paged_attention(q, kc, vc, tables, starts, at.int().cuda(), **common)
        torch.cuda.synchronize()
        out = ops.paged_attention(q, kc, vc, tables, starts, ops.argmax_rows(marked), **common)
        assert torch.equal(out, ref), i


@pytest.mark.parametrize("summed", [False, True])
def test_portions_launch_without_tiles_keeps_the_order_of_kernels(ops, monkeypatch, summed):
    """A step of short requests whose lengths the host does not tell: the portions' kernel is launched first and finds no
    tile of its own. The decode kernel behind it still comes after what makes the queries, a product here."""
    import atomserve_b200.ops.attention as attention

    monkeypatch.setattr(attention, "MIXED_OVERLAP", False)  # both kernels on one stream
    lens, q_lens, H, KV, hd = [700, 1200, 64, 2000] * 8, [1, 8, 2, 1] * 8, 8, 2, 128
    dev, dense, qs = paged_setup(lens, q_lens, H, KV, hd, 16, torch.bfloat16)
    T, parts = sum(q_lens), KV if summed else 1
    g = torch.Generator().manual_seed(2)
    x = torch.randn(T, 4096, generator=g).bfloat16().cuda()
    w = (torch.randn(H * parts * hd, 4096, generator=g) / 64).bfloat16().cuda()

    def queries():
        q = ops.linear(x, w)
        return q.view(T, H, KV, hd) if summed else q.view(T, H, hd)

    common = dict(dev, num_requests=len(lens), max_context=max(lens), window=None, scale=hd**-0.5)
    common["q"] = queries()
    torch.cuda.synchronize()
    ref = ops.paged_attention(**common)
    known = ops.paged_attention(**common, host_q_lens=q_lens)
    torch.cuda.synchronize()
    assert torch.allclose(ref.float(), known.float(), atol=2e-2, rtol=2e-2)  # (shares of a row's keys may be others)
    for _ in range(20):
        common["q"] = queries()
        assert torch.equal(ops.paged_attention(**common), ref)


@pytest.mark.parametrize("lens,q_lens,H,KV,window", [
    ([700, 40, 65], [300, 40, 9], 32, 8, None),     # tiles that see fewer key tiles than there are parts, beside long ones
    ([1500, 90], [130, 64], 10, 2, None),           # padding rows in every tile, an odd number of key tiles
    ([1200, 300], [200, 100], 16, 1, 150),          # a window: parts in which a row sees nothing
])  # fmt: skip
@pytest.mark.parametrize("parts", [1, 2, 4])
@pytest.mark.parametrize("with_sink,chunk,softcap", [(False, None, None), (True, None, None), (False, 256, None), (True, 333, 2.0)])
def test_prefill_attention_tcgen05_in_parts(ops, monkeypatch, lens, q_lens, H, KV, window, parts, with_sink, chunk, softcap):
    """Prompt portions whose key tiles are divided among the blocks of a cluster, against the general kernel in float32."""
    import atomserve_b200.ops.attention as attention
    from atomserve_b200.ops.linear import check_gemm_status

    dev, dense, qs = paged_setup(lens, q_lens, H, KV, 128, 16, torch.bfloat16)
    sink = torch.linspace(-2, 3, H, device="cuda") if with_sink else None
    common = dict(num_requests=len(lens), max_context=max(lens), window=window, scale=128**-0.5, host_q_lens=q_lens, sink=sink,
                  chunk=chunk, softcap=softcap)  # fmt: skip
    wide = {k: (v.float() if v.dtype == torch.bfloat16 else v) for k, v in dev.items()}
    ref = ops.paged_attention(**wide, **common, generic=True)
    monkeypatch.setattr(attention, "plan_portion_parts", lambda *a: parts)
    out = ops.paged_attention(**dev, **common)
    check_gemm_status()
    # bfloat16 values and probabilities: 2^-8 of values of size one, a few times over
    assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2), float((out.float() - ref).abs().max())


@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("where", [5, 700, 1500])
@pytest.mark.parametrize("q_lens,shares", [([1, 1, 1], 0), ([1, 1, 1], 2), ([1, 1, 1], 17), ([200, 90, 64], 1), ([200, 90, 64], 2), ([200, 90, 64], 4)])
@pytest.mark.parametrize("with_sink", [False, True])
def test_a_key_that_is_not_finite_shows_however_keys_are_shared(ops, monkeypatch, bad, where, q_lens, shares, with_sink):
    """One key of request 0 (kv head 1) with a NaN or an infinity: exactly the outputs that see it are NaN, whether a row's
    keys are one walk or shares that are merged (the decode kernel's ranges, the parts of a portion)."""
    import atomserve_b200.ops.attention as attention

    lens, H, KV, hd, bs = [1600, 300, 700], 8, 2, 128, 16
    dev, dense, qs = paged_setup(lens, q_lens, H, KV, hd, bs, torch.bfloat16)
    dev["k_cache"][dev["block_tables"][0, where // bs].long(), 1, where % bs] = bad
    sink = torch.linspace(-2, 3, H, device="cuda") if with_sink else None
    monkeypatch.setattr(attention, "plan_decode_ranges", lambda *a: shares)
    monkeypatch.setattr(attention, "plan_portion_parts", lambda *a: shares)
    out = ops.paged_attention(**dev, num_requests=3, max_context=max(lens), window=None, scale=hd**-0.5, host_q_lens=q_lens, sink=sink)
    sees = torch.arange(lens[0] - q_lens[0], lens[0]) >= where  # by position, of request 0's rows
    expect = torch.zeros(sum(q_lens), H, dtype=torch.bool)
    expect[: q_lens[0], H // KV :] = sees[:, None]
    got = torch.isnan(out).cpu()
    assert torch.equal(got.all(-1), expect) and torch.equal(got.any(-1), expect)


@pytest.mark.parametrize("tokens", [32, 64, 96, 160, 224, 256])
@pytest.mark.parametrize("M,N,K", [(300, 512, 256), (33, 130, 72), (257, 4104, 520), (160, 6144, 4160), (5, 24576, 1024), (70, 256, 64),
                                   (131, 2000, 12288), (513, 1000, 4160)])  # fmt: skip
def test_gemm_tcgen05_on_pairs_of_sms_swapped(ops, M, N, K, tokens):
    """The pair form with its operands swapped (tiles of 256 weight rows by 32 to 256 tokens), forced: every epilogue against
    float64; tokens, weight rows and K that end inside a tile, one tile, more tiles than pairs, tiles cut along K."""
    from atomserve_b200.ops.linear import check_gemm_status, gemm_tcgen05, gemm_tune

    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).bfloat16().cuda()
    res = torch.randn(M, N, generator=g).bfloat16().cuda()
    ref = x.double().cpu() @ w.double().cpu().T
    gemm_tune(3, tokens)
    try:
        full = gemm_tcgen05(x, w, None, torch.float32)
        plain_out = gemm_tcgen05(x, w, None, torch.bfloat16)
        with_res = gemm_tcgen05(x, w, res, torch.bfloat16)
        squared = gemm_tcgen05(x, w, None, torch.bfloat16, relu2=True)
        fused = gemm_tcgen05(x, w, None, torch.bfloat16, swiglu=True)
        again = gemm_tcgen05(x, w, None, torch.float32)
        gemm_tune(3, tokens, cut_last_round=False)
        uncut = gemm_tcgen05(x, w, None, torch.float32)
    finally:
        gemm_tune()
    check_gemm_status()
    assert torch.allclose(uncut, full, atol=1e-4, rtol=1e-4)  # cut or whole, the same products are added, in another order
    assert torch.allclose(full.double().cpu(), ref, atol=2e-3, rtol=1e-3), float((full.double().cpu() - ref).abs().max())
    assert torch.equal(again, full)
    assert torch.allclose(plain_out.double().cpu(), ref, atol=3e-2, rtol=2e-2)
    assert torch.allclose(with_res.double().cpu(), ref + res.double().cpu(), atol=3e-2, rtol=2e-2)
    assert torch.allclose(squared.double().cpu(), ref.clamp_min(0) ** 2, atol=3e-2, rtol=2e-2)
    gate, up = ref[:, 0::2], ref[:, 1::2]
    assert torch.allclose(fused.double().cpu(), gate / (1 + torch.exp(-gate)) * up, atol=3e-2, rtol=3e-2)
