"""GPU parity of the dense projections (tcgen05 GEMM for bf16/fp16, FFMA for
fp32) through the C ABI, against a plain fp32 torch matmul of the same operands
and against the CPU oracle for the fused epilogues."""
import pytest
import torch

from helpers import rel_err
from oracle import tp_layer_oracle as O

pytestmark = pytest.mark.gpu

GEMM_TOL = {torch.float32: 2e-5, torch.bfloat16: 1e-2, torch.float16: 2e-3}


def _rand(shape, dtype, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype)


# Per-rank shapes of the 70B-shaped layer at TP=8 (hidden 8192, 64 q / 8 kv heads, intermediate 28672;
# T = 512): qkv N=1280, o_proj K=1024, gate_up N=7168 (d=3584), down K=3584.
def test_70b_shaped_tp8_shard_projections():
    from sarathi_serve_b200 import dense_ops
    T, H = 512, 8192
    dtype = torch.bfloat16
    x = _rand((T, H), dtype, 11)
    # qkv + rotary: 8 q heads + 1 k head rotated, 1 v head untouched
    wqkv = _rand((1280, H), dtype, 12, 0.02)
    pos = torch.arange(T, dtype=torch.int64) * 5 % 4096
    cache = O.cos_sin_cache(128, 128, 8192, 500000.0, dtype)
    ref = (x.float() @ wqkv.float().t()).to(dtype)
    q, k = ref[:, :1024].clone(), ref[:, 1024:1152].clone()
    O.rotary_embedding(pos, q, k, 128, cache, True)
    out = dense_ops.linear_rotary(x.cuda(), wqkv.cuda(), pos.cuda(), cache.cuda(), 128, 1152, True)
    _check_status()
    assert rel_err(out[:, :1024].float().cpu(), q.float()) <= 2e-2
    assert rel_err(out[:, 1024:1152].float().cpu(), k.float()) <= 2e-2
    assert rel_err(out[:, 1152:].float().cpu(), ref[:, 1152:].float()) <= 2e-2
    # gate_up + SiLU*mul
    wgu = _rand((7168, H), dtype, 13, 0.02)
    gu = (x.float() @ wgu.float().t()).to(dtype)
    act_ref = O.silu_and_mul(gu)
    act = dense_ops.linear_silu_mul(x.cuda(), wgu.cuda())
    _check_status()
    assert rel_err(act.float().cpu(), act_ref.float()) <= 2e-2
    # o_proj / down shards (K = 1024, 3584), output rows of 16 KiB
    for K, seed in ((1024, 14), (3584, 15)):
        a, w = _rand((T, K), dtype, seed), _rand((H, K), dtype, seed + 10, 0.02)
        y = dense_ops.linear(a.cuda(), w.cuda())
        _check_status()
        assert rel_err(y.float().cpu(), a.float() @ w.float().t()) <= 2e-2


def _check_status():
    from sarathi_serve_b200 import dense_ops
    dense_ops.check_status(torch.device("cuda", torch.cuda.current_device()))


# tile configuration = BN + 1000*MI + 100000*splitK (0 = chosen by the library)
TILE_CFGS = [0, 64, 96, 128, 160, 224, 256, 2064, 2128, 2256, 301128, 402256, 1602128, 200032,
             3064, 3128, 3192, 3256, 203256, 503128, 4064, 4128, 4256, 304256,  # 3xxx/4xxx = CTA pairs (cta_group::2)
             205256, 205128, 405128, 205064, 405064, 405192]  # 5xxx = a cluster of 2 / 4 CTA pairs splits the K of every tile


def _skip_unless_planned(epi, T, N, K, cfg, head_size=128):
    """Cluster K-split configurations are only accepted for problems with few tiles (one cluster per tile)."""
    from sarathi_serve_b200 import dense_ops
    if (cfg // 1000) % 100 == 5:
        try:
            dense_ops.gemm_plan(epi, T, N, K, head_size, cfg)
        except RuntimeError:
            pytest.skip("this problem does not fit the cluster K-split configuration")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("tile_n", TILE_CFGS)
@pytest.mark.parametrize("T,N,K", [(128, 128, 64), (128, 256, 128), (512, 768, 4096), (288, 768, 1024), (1, 256, 512),
                                   (65, 200, 264), (300, 1000, 1000), (512, 6144, 512), (1024, 8, 4096)])
def test_linear(dtype, tile_n, T, N, K):
    from sarathi_serve_b200 import dense_ops
    if dtype == torch.float32 and tile_n not in (0,):
        pytest.skip("tile shape applies to the tensor-core path only")
    if tile_n // 100000 > (K + 63) // 64:
        pytest.skip("more splits than k-blocks")
    _skip_unless_planned(0, T, N, K, tile_n)
    x, w = _rand((T, K), dtype, T + N + K), _rand((N, K), dtype, 7 * N + K, 0.05)
    b = _rand((N,), dtype, 3)
    ref = x.float().cuda() @ w.float().cuda().t()
    out = dense_ops.linear(x.cuda(), w.cuda(), tile_n=tile_n)
    _check_status()
    assert rel_err(out.float(), ref) <= GEMM_TOL[dtype]
    outb = dense_ops.linear(x.cuda(), w.cuda(), b.cuda(), tile_n=tile_n)
    assert rel_err(outb.float(), ref + b.float().cuda()) <= GEMM_TOL[dtype]


# tile edges of the fp32 kernel (32 / 64 rows, 128 columns, 16 k), K cut over 1..8 CTAs, rows that are not 16-byte aligned
@pytest.mark.parametrize("T,N,K", [(1, 1, 1), (32, 128, 4096), (33, 129, 1023), (31, 5, 64), (64, 640, 68), (65, 257, 2816),
                                   (288, 1536, 1024), (512, 128, 130)])
@pytest.mark.parametrize("pad", [0, 3])
def test_linear_f32_tiles(T, N, K, pad):
    from sarathi_serve_b200 import dense_ops
    x = _rand((T, K + pad), torch.float32, T + N + K).cuda()[:, pad:]
    w = _rand((N, K + pad), torch.float32, 7 * N + K).cuda()[:, pad:]
    b = _rand((N,), torch.float32, 3).cuda()
    out = torch.full((T, N + pad), 7.0, device="cuda")
    dense_ops.linear(x, w, b, out=out[:, pad:])
    ref = x.double() @ w.double().t() + b.double()
    # K products and K + 9 sums, each rounded once to fp32: |err| <= (K + 10) * 2^-24 * sum |x||w|; random signs leave
    # about the square root of that many roundings
    bound = 4 * (K + 10) ** 0.5 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t() + b.double().abs())
    assert bool(((out[:, pad:].double() - ref).abs() <= bound).all())
    assert pad == 0 or bool((out[:, :pad] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tile_n", [0, 128, 3256, 203128, 2064, 205256, 405128])
@pytest.mark.parametrize("T,N,K", [(512, 4096, 512), (65, 200, 264), (300, 1000, 1000), (1, 256, 512)])
def test_linear_with_residual_in_the_epilogue(dtype, tile_n, T, N, K):
    """out = residual + round(x w^T + b): the reference's `hidden_states = residual + hidden_states` after a
    row-parallel projection (models/llama.py:248,254) fused into the plain GEMM (what runs at TP = 1)."""
    from oracle import tp_layer_oracle as O
    from sarathi_serve_b200 import dense_ops
    if tile_n // 100000 > (K + 63) // 64:
        pytest.skip("more splits than k-blocks")
    _skip_unless_planned(0, T, N, K, tile_n)
    x, w = _rand((T, K), dtype, T + N + K), _rand((N, K), dtype, 7 * N + K, 0.05)
    b, r = _rand((N,), dtype, 3), _rand((T, N), dtype, 4)
    ref = r + O.linear(x.float(), w.float(), b.float()).to(dtype)
    out = dense_ops.linear(x.cuda(), w.cuda(), b.cuda(), tile_n=tile_n, residual=r.cuda())
    _check_status()
    assert rel_err(out.float(), ref.float()) <= GEMM_TOL[dtype]
    # strided residual view and a caller-provided output
    big = torch.zeros(T, N + 64, dtype=dtype, device="cuda")
    big[:, 32:32 + N] = r.cuda()
    out2 = torch.empty(T, N, dtype=dtype, device="cuda")
    dense_ops.linear(x.cuda(), w.cuda(), b.cuda(), out=out2, tile_n=tile_n, residual=big[:, 32:32 + N])
    assert torch.equal(out2, out)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_linear_strided_operands(dtype):
    """A and the output may be row-strided views (q view of the fused qkv buffer feeding o_proj)."""
    from sarathi_serve_b200 import dense_ops
    big = _rand((130, 1536), dtype, 1).cuda()
    x = big[:, 256:256 + 512]  # row stride 1536, 16-byte aligned start
    w = _rand((384, 512), dtype, 2, 0.05).cuda()
    outbuf = torch.zeros(130, 1024, dtype=dtype, device="cuda")
    out = outbuf[:, 128:128 + 384]
    dense_ops.linear(x, w, out=out)
    _check_status()
    assert rel_err(out.float(), x.float() @ w.float().t()) <= GEMM_TOL[dtype]
    assert torch.all(outbuf[:, :128] == 0) and torch.all(outbuf[:, 512:] == 0)


def test_linear_rejects_misaligned_stride():
    from sarathi_serve_b200 import dense_ops
    x = torch.randn(16, 100, dtype=torch.bfloat16, device="cuda")[:, :68]  # 68*2 bytes rows of a 100-wide buffer
    w = torch.randn(32, 68, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(RuntimeError):
        dense_ops.linear(x[:, 1:65], w[:, :64].contiguous())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("neox", [True, False])
@pytest.mark.parametrize("tile_n", [0, 256, 2256, 401256, 302256, 3256, 303256, 4256, 204128,
                                    # 64-column tiles: for NeoX heads wider than 64 a tile holds 32 + 32 columns of
                                    # the two halves of a head, so that every rotation pair sits in one accumulator
                                    64, 2064, 3064, 4064, 303064, 600064,
                                    205128, 405128, 205064, 405256])
@pytest.mark.parametrize("T,nq,nkv,hd,K", [(512, 4, 1, 128, 4096), (288, 8, 2, 64, 1024), (65, 2, 2, 128, 512),
                                           (7, 1, 1, 256, 256)])
def test_linear_rotary(dtype, neox, tile_n, T, nq, nkv, hd, K):
    from sarathi_serve_b200 import dense_ops
    N = (nq + 2 * nkv) * hd
    x, w = _rand((T, K), dtype, T + K), _rand((N, K), dtype, N, 0.03)
    g = torch.Generator().manual_seed(5)
    pos = torch.randint(0, 2048, (T,), generator=g, dtype=torch.int64)
    cache = O.cos_sin_cache(hd, hd, 2048, 10000.0, dtype)
    split_head = neox and tile_n % 1000 == 64 and hd > 64
    if tile_n // 100000 > (K + 63) // 64 or (tile_n and (tile_n % 1000) % hd and not split_head):
        pytest.skip("tile configuration does not fit this case")
    _skip_unless_planned(1, T, (nq + 2 * nkv) * hd, K, tile_n, hd)
    out = dense_ops.linear_rotary(x.cuda(), w.cuda(), pos.cuda(), cache.cuda(), hd, (nq + nkv) * hd, neox,
                                  tile_n=tile_n)
    _check_status()
    # oracle: GEMM rounded to the dtype (GPU fp32 matmul of the same operands), then the rotary restatement
    ref = (x.float().cuda() @ w.float().cuda().t()).to(dtype).cpu()
    q, k, _ = ref.split([nq * hd, nkv * hd, nkv * hd], dim=-1)
    O.rotary_embedding(pos, q, k, hd, cache, neox)
    assert rel_err(out, ref) <= GEMM_TOL[dtype]
    # v columns are a plain GEMM
    assert rel_err(out[:, (nq + nkv) * hd:], ref[:, (nq + nkv) * hd:]) <= GEMM_TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tile_n", [0, 64, 128, 192, 256, 2128, 2256, 501256, 402128, 3064, 3128, 3256, 403256, 4128, 4256, 304256,
                                    205256, 405128, 205064])
@pytest.mark.parametrize("T,d,K", [(512, 1792, 4096), (288, 1408, 1024), (65, 96, 512), (1, 64, 64)])
def test_linear_silu_mul(dtype, tile_n, T, d, K):
    from sarathi_serve_b200 import dense_ops
    if tile_n // 100000 > (K + 63) // 64:
        pytest.skip("more splits than k-blocks")
    _skip_unless_planned(2, T, 2 * d, K, tile_n)
    x, w = _rand((T, K), dtype, T + K), _rand((2 * d, K), dtype, d, 0.05)
    out = dense_ops.linear_silu_mul(x.cuda(), w.cuda(), tile_n=tile_n)
    _check_status()
    gate_up = (x.float().cuda() @ w.float().cuda().t()).to(dtype).cpu()
    ref = O.silu_and_mul(gate_up)
    assert out.shape == (T, d)
    assert rel_err(out, ref) <= 2e-2


# Small batches run on a kernel of their own (tokens as the N side of the MMA, K cut over a cluster): edges of its token
# granules (8, 16, 64), of its 128-column tiles, of a head's halves, one and many k-blocks, and more tiles than SMs.
def _bf_bound(ref64, absum, K, dtype):
    """One rounding of the result to the 16-bit type plus K + 64 fp32 roundings of products and sums."""
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    return u * ref64.abs() + (K + 64) * 2.0 ** -24 * absum + 1e-7


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,N,K", [(1, 128, 64), (8, 4096, 512), (9, 200, 264), (16, 384, 1000), (17, 17, 4096), (63, 768, 4096),
                                   (64, 130, 1792), (5, 20000, 128), (64, 19072, 64), (65, 256, 512)])
def test_linear_small_batch(dtype, T, N, K):
    from sarathi_serve_b200 import dense_ops
    x, w = _rand((T, K + 64), dtype, T + N + K).cuda()[:, 64:], _rand((N, K), dtype, 7 * N + K, 0.05).cuda()
    b, r = _rand((N,), dtype, 3).cuda(), _rand((T, N + 3), dtype, 4).cuda()[:, 3:]
    out = torch.full((T, N + 1), 7.0, dtype=dtype, device="cuda")
    dense_ops.linear(x, w, out=out[:, 1:])
    _check_status()
    ref, absum = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert bool(((out[:, 1:].double() - ref).abs() <= _bf_bound(ref, absum, K, dtype)).all())
    assert bool((out[:, 0] == 7.0).all())
    # bias and residual: the same sums through the other kernel, rounded at the same places
    got = dense_ops.linear(x, w, b, residual=r)
    want = dense_ops.linear(x, w, b, residual=r, tile_n=128)
    assert rel_err(got.float(), want.float()) <= GEMM_TOL[dtype]
    assert rel_err(got.float(), r.double() + (ref + b.double()).to(dtype).double()) <= GEMM_TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,d,K", [(1, 64, 64), (8, 14336, 256), (16, 96, 520), (31, 1792, 4096), (64, 200, 512)])
def test_linear_silu_mul_small_batch(dtype, T, d, K):
    from sarathi_serve_b200 import dense_ops
    x, w = _rand((T, K), dtype, T + K), _rand((2 * d, K), dtype, d, 0.05)
    out = dense_ops.linear_silu_mul(x.cuda(), w.cuda())
    _check_status()
    ref = O.silu_and_mul((x.float().cuda() @ w.float().cuda().t()).to(dtype).cpu())
    assert rel_err(out, ref) <= 2e-2
    assert rel_err(out, dense_ops.linear_silu_mul(x.cuda(), w.cuda(), tile_n=128)) <= 2e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,nq,nkv,hd,K", [(1, 1, 1, 64, 64), (8, 4, 1, 128, 4096), (17, 3, 1, 256, 264), (64, 5, 2, 64, 1024),
                                           (61, 32, 8, 128, 512)])
def test_linear_rotary_small_batch(dtype, T, nq, nkv, hd, K):
    """Against the general kernel (its tiles hold whole heads), with the append to the paged cache."""
    from sarathi_serve_b200 import dense_ops
    N, page = (nq + 2 * nkv) * hd, 16
    x, w = _rand((T, K), dtype, T + K).cuda(), _rand((N, K), dtype, N, 0.03).cuda()
    g = torch.Generator().manual_seed(5)
    pos = torch.randint(0, 2048, (T,), generator=g).cuda()
    cs = O.cos_sin_cache(hd, hd, 2048, 10000.0, dtype).cuda()
    res = []
    for cfg in (0, 256):
        cache = torch.zeros((T + page - 1) // page + 1, 2, page, nkv, hd, dtype=dtype, device="cuda")
        # distinct slots only: tokens that share one would race
        s = torch.full((T,), -1, dtype=torch.int64, device="cuda")
        live = torch.arange(T, device="cuda") % 5 != 0
        s[live] = (torch.arange(T, device="cuda") // page * 2 * page + torch.arange(T, device="cuda") % page)[live]
        out = dense_ops.linear_rotary(x, w, pos, cs, hd, (nq + nkv) * hd, True, tile_n=cfg, kv_cache=cache, kv_slots=s,
                                      num_kv_heads=nkv)
        _check_status()
        res.append((out, cache))
        k, v = out[:, nq * hd:(nq + nkv) * hd], out[:, (nq + nkv) * hd:]
        flat = cache.view(-1, nkv * hd)
        assert torch.equal(flat[s[live]], k[live]) and torch.equal(flat[s[live] + page], v[live])
        assert int((flat.abs().sum(1) > 0).sum()) == 2 * int(live.sum())
    assert rel_err(res[0][0], res[1][0]) <= GEMM_TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,N,K", [(1, 1, 8), (3, 8, 4096), (297, 8, 264), (1024, 8, 4096), (24, 16, 2048), (300, 9, 2056)])
def test_linear_few_columns(dtype, T, N, K):
    from sarathi_serve_b200 import dense_ops
    x, w = _rand((T, K + 8), dtype, T + N + K).cuda()[:, 8:], _rand((N, K), dtype, 7 * N + K, 0.05).cuda()
    b, r = _rand((N,), dtype, 3).cuda(), _rand((T, N), dtype, 4).cuda()
    out = dense_ops.linear(x, w)
    ref, absum = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert bool(((out.double() - ref).abs() <= _bf_bound(ref, absum, K, dtype)).all())
    got = dense_ops.linear(x, w, b, residual=r)
    assert rel_err(got.float(), r.double() + (ref + b.double()).to(dtype).double()) <= GEMM_TOL[dtype]


# The same kernel on larger, ragged batches: token tiles of 16..176 (the tokens are spread evenly over the tiles), one and two
# accumulators, K over a cluster.  More than one round of tiles only for 6016 and 7064 with 513 tokens, both on two sets of
# accumulators; the other rounds: test_swapped_tiles_over_several_rounds.
@pytest.mark.parametrize("cfg", [6016, 6112, 6128, 6256, 7064, 7256, 206064, 807032, 306176])
@pytest.mark.parametrize("T,N,K", [(65, 256, 512), (129, 200, 1000), (300, 1000, 512), (513, 4096, 576)])
def test_linear_swapped_tiles(cfg, T, N, K):
    from sarathi_serve_b200 import dense_ops
    p = dense_ops.gemm_launch(0, T, N, K, tile_cfg=cfg)
    assert p["kernel"] == "swapped" and p["k_parts"] == max(1, cfg // 100000)
    x, w = _rand((T, K), torch.bfloat16, T + N).cuda(), _rand((N, K), torch.bfloat16, N + K, 0.05).cuda()
    b, r = _rand((N,), torch.bfloat16, 3).cuda(), _rand((T, N), torch.bfloat16, 4).cuda()
    out = dense_ops.linear(x, w, tile_n=cfg)
    _check_status()
    ref, absum = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert bool(((out.double() - ref).abs() <= _bf_bound(ref, absum, K, torch.bfloat16)).all())
    got = dense_ops.linear(x, w, b, tile_n=cfg, residual=r)
    assert rel_err(got.float(), r.double() + (ref + b.double()).to(torch.bfloat16).double()) <= GEMM_TOL[torch.bfloat16]


@pytest.mark.parametrize("cfg", [6048, 6112, 6256, 206096])
@pytest.mark.parametrize("T,nq,nkv,hd", [(100, 2, 1, 64), (300, 4, 2, 128), (131, 1, 1, 256)])
def test_linear_rotary_and_silu_swapped_tiles(cfg, T, nq, nkv, hd):
    from sarathi_serve_b200 import dense_ops
    N, K = (nq + 2 * nkv) * hd, 320
    assert all(dense_ops.gemm_launch(epi, T, N, K, hd, cfg)["kernel"] == "swapped" for epi in (1, 2))
    x, w = _rand((T, K), torch.float16, T).cuda(), _rand((N, K), torch.float16, N, 0.05).cuda()
    pos = torch.randint(0, 2048, (T,), generator=torch.Generator().manual_seed(5)).cuda()
    cs = O.cos_sin_cache(hd, hd, 2048, 10000.0, torch.float16).cuda()
    caches = [torch.zeros(T, 2, 1, nkv, hd, dtype=torch.float16, device="cuda") for _ in range(2)]
    slots = torch.arange(T, device="cuda").flip(0) * 2
    outs = [dense_ops.linear_rotary(x, w, pos, cs, hd, (nq + nkv) * hd, True, tile_n=c, kv_cache=kc, kv_slots=slots,
                                    num_kv_heads=nkv) for c, kc in zip((cfg, 256), caches)]
    _check_status()
    assert rel_err(outs[0], outs[1]) <= GEMM_TOL[torch.float16] and rel_err(caches[0], caches[1]) <= GEMM_TOL[torch.float16]
    assert torch.equal(caches[0].view(T, 2, -1)[slots // 2, 1], outs[0][:, (nq + nkv) * hd:])
    acts = [dense_ops.linear_silu_mul(x, w, tile_n=c) for c in (cfg, 128)]
    _check_status()
    assert rel_err(acts[0], acts[1]) <= 2e-2


# Several rounds of tiles per CTA, on one set of accumulators (a tile is finished before the next one's MMAs) and on two (its
# epilogue under the next tile's loop), three and more uses of a set; the largest token tiles.
@pytest.mark.parametrize("epi,T,cols,K,cfg,tokens,sets,rounds", [
    ("silu", 300, 14336, 128, 6160, 160, 1, 2), ("silu", 800, 14336, 64, 6160, 160, 1, 4), ("silu", 896, 14336, 64, 6128, 128, 2, 6),
    ("silu", 16, 19100, 64, 6016, 16, 2, 2), ("silu", 512, 200, 264, 6256, 256, 1, 1), ("silu", 200, 14336, 192, 6208, 208, 1, 1),
    ("store", 800, 25600, 64, 6160, 160, 1, 4), ("store", 1120, 15300, 72, 6112, 112, 2, 5), ("store", 512, 1000, 520, 6256, 256, 1, 1),
    ("store", 2048, 8000, 64, 7256, 256, 2, 4), ("store", 200, 300, 264, 7208, 208, 1, 1),
    ("rotary", 800, 15360, 64, 6160, 160, 1, 3), ("rotary", 1120, 15360, 64, 6112, 112, 2, 5), ("rotary", 512, 768, 320, 6256, 256, 1, 1),
    ("rotary", 200, 1024, 264, 6208, 208, 1, 1)])
def test_swapped_tiles_over_several_rounds(epi, T, cols, K, cfg, tokens, sets, rounds):
    from sarathi_serve_b200 import dense_ops
    dtype, hd, u = torch.float16, 128, 2.0 ** -11
    N = 2 * cols if epi == "silu" else cols
    p = dense_ops.gemm_launch({"store": 0, "rotary": 1, "silu": 2}[epi], T, N, K, hd, cfg)
    assert (p["kernel"], p["tokens"], p["accumulator_sets"], p["rounds"]) == ("swapped", tokens, sets, rounds)
    x, w = _rand((T, K), dtype, T + K).cuda(), _rand((N, K), dtype, N + K, 0.1).cuda()
    y, absum = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    sums = (K + 64) * 2.0 ** -24 * absum  # products and sums in fp32
    if epi == "store":
        out = dense_ops.linear(x, w, tile_n=cfg)
        _check_status()
        assert bool(((out.double() - y).abs() <= _bf_bound(y, absum, K, dtype)).all())
        return
    if epi == "silu":
        out = dense_ops.linear_silu_mul(x, w, tile_n=cfg)
        _check_status()
        g, up = y[:, :cols], y[:, cols:]
        f = g * torch.sigmoid(g)
        # gate rounded before silu (slope at most 1.1), silu, up and the product rounded; 5 % for the terms of higher order
        bound = 1.1 * (u * g.abs() + sums[:, :cols]) * up.abs() + f.abs() * (3.2 * u * up.abs() + sums[:, cols:])
        assert bool(((out.double() - f * up).abs() <= 1.05 * bound + 1e-6).all())
        return
    heads = cols // hd
    nkv = heads // 6
    rot, page = (heads - nkv) * hd, 16
    pos = torch.randint(0, 2048, (T,), generator=torch.Generator().manual_seed(5)).cuda()
    cs = O.cos_sin_cache(hd, hd, 2048, 10000.0, dtype).cuda()
    cache = torch.zeros((T + page - 1) // page, 2, page, nkv, hd, dtype=dtype, device="cuda")
    t = torch.arange(T, device="cuda")
    slots = t // page * 2 * page + t % page
    out = dense_ops.linear_rotary(x, w, pos, cs, hd, rot, True, tile_n=cfg, kv_cache=cache, kv_slots=slots, num_kv_heads=nkv)
    _check_status()
    c, s = cs[pos].double()[:, None, :hd // 2], cs[pos].double()[:, None, hd // 2:]

    def halves(m):
        m = m[:, :rot].view(T, -1, hd)
        return m[..., :hd // 2], m[..., hd // 2:]
    (a, b), (ea, eb) = halves(y), halves(sums)
    want = torch.cat([a * c - b * s, b * c + a * s], -1).view(T, rot)
    # both inputs, both products and the result rounded
    ra, rb = 2 * u * a.abs() + ea, 2 * u * b.abs() + eb
    bound = torch.cat([ra * c.abs() + rb * s.abs(), rb * c.abs() + ra * s.abs()], -1).view(T, rot) + u * want.abs()
    assert bool(((out[:, :rot].double() - want).abs() <= 1.05 * bound + 1e-6).all())
    assert bool(((out[:, rot:].double() - y[:, rot:]).abs() <= _bf_bound(y, absum, K, dtype)[:, rot:]).all())
    flat, kv = cache.view(-1, nkv * hd), nkv * hd
    assert torch.equal(flat[slots], out[:, rot - kv:rot]) and torch.equal(flat[slots + page], out[:, rot:rot + kv])


# Explicit configurations that do not fit are refused, not run as something else: too few and too many tokens a tile, more
# parts than k-blocks, more than eight, an exchange larger than the ring, two accumulators' epilogue on one.
@pytest.mark.parametrize("epi,cfg", [("store", 6008), ("store", 6300), ("store", 806064), ("store", 906064), ("store", 206256),
                                     ("silu", 7064)])
def test_swapped_tiles_that_do_not_fit_are_refused(epi, cfg):
    from sarathi_serve_b200 import dense_ops
    x, w = _rand((256, 256), torch.bfloat16, 1).cuda(), _rand((512, 256), torch.bfloat16, 2, 0.05).cuda()
    with pytest.raises(RuntimeError, match="no GEMM tile shape fits"):
        dense_ops.linear(x, w, tile_n=cfg) if epi == "store" else dense_ops.linear_silu_mul(x, w, tile_n=cfg)


# The library's own choice on both sides of its rule: K cut over clusters that all run at once, whole tiles, CTA pairs.
@pytest.mark.parametrize("T", [33, 65, 130, 270, 513])
@pytest.mark.parametrize("nq,nkv", [(4, 1), (8, 2), (16, 4)])
def test_linear_rotary_and_silu_chosen_tiles(T, nq, nkv):
    from sarathi_serve_b200 import dense_ops
    hd, K = 128, 2048
    N = (nq + 2 * nkv) * hd
    x, w = _rand((T, K), torch.float16, T).cuda(), _rand((N, K), torch.float16, N, 0.05).cuda()
    pos = torch.randint(0, 2048, (T,), generator=torch.Generator().manual_seed(6)).cuda()
    cs = O.cos_sin_cache(hd, hd, 2048, 10000.0, torch.float16).cuda()
    outs = [dense_ops.linear_rotary(x, w, pos, cs, hd, (nq + nkv) * hd, True, tile_n=c) for c in (0, 128)]
    acts = [dense_ops.linear_silu_mul(x, w, tile_n=c) for c in (0, 128)]
    _check_status()
    assert rel_err(outs[0], outs[1]) <= GEMM_TOL[torch.float16]
    assert rel_err(acts[0], acts[1]) <= 2e-2


# The last, partial 128-row block of A is loaded by a shorter box, blocks without rows not at all.
@pytest.mark.parametrize("tile_n", [128, 2064, 3128, 4064, 203064, 301128, 205064])
@pytest.mark.parametrize("T", [1, 8, 127, 129, 255, 257, 385])
def test_linear_partial_row_blocks(tile_n, T):
    from sarathi_serve_b200 import dense_ops
    K, N = 512, 192
    _skip_unless_planned(0, T, N, K, tile_n)
    x, w = _rand((T, K), torch.bfloat16, T).cuda(), _rand((N, K), torch.bfloat16, 9, 0.05).cuda()
    out = dense_ops.linear(x, w, tile_n=tile_n)
    _check_status()
    ref, absum = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert bool(((out.double() - ref).abs() <= _bf_bound(ref, absum, K, torch.bfloat16)).all())


def test_gemm_linearity_full_size():
    """Size-independent property at the headline shapes: (a*x) W^T == a * (x W^T) for a power of two."""
    from sarathi_serve_b200 import dense_ops
    x = _rand((512, 4096), torch.bfloat16, 1).cuda()
    w = _rand((3584 * 2, 4096), torch.bfloat16, 2, 0.02).cuda()
    y1 = dense_ops.linear(x, w)
    y2 = dense_ops.linear(x * 4, w)
    _check_status()
    assert torch.equal(y1 * 4, y2)


def test_mma_rate_diagnostic_runs_and_orders_the_two_modes():
    """The planner's two constants, re-measured: a CTA pair completes a 256-row MMA of N = 128 in fewer clocks than
    one CTA needs for its 128-row MMA, and N = 256 on a pair takes about twice as long as N = 128."""
    from sarathi_serve_b200 import mma_rate
    one = mma_rate.measure(False, 128, iters=256)
    pair128 = mma_rate.measure(True, 128, iters=256)
    pair256 = mma_rate.measure(True, 256, iters=256)
    for r in (one, pair128, pair256):
        assert 8 < r["clk_per_mma_complete"] < 2000, r
    assert pair128["clk_per_mma_complete"] < one["clk_per_mma_complete"]
    assert 1.5 < pair256["clk_per_mma_complete"] / pair128["clk_per_mma_complete"] < 2.5
