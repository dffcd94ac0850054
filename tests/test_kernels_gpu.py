"""CUDA kernels against plain PyTorch fp32 references (single GPU; peers emulated by local buffers)."""
import math
import os

import pytest
import torch

pytestmark = pytest.mark.gpu

# The fused GEMMs can start their walk over the owners at the calling rank's own rows (off by default, read once per
# process).  Switched on here so that the emulated-rank cases below, which pass non-zero positions, cover the rotated
# tile, fetch and k orders; position 0 and the other test files cover the unrotated order.
os.environ.setdefault("ODC_GEMM_ROTATE", "2")


@pytest.fixture(scope="module")
def ext():
    from odc_b200 import _ext
    return _ext.load()


def _table(tensors):
    return torch.tensor([t.data_ptr() for t in tensors], dtype=torch.int64, device="cuda")


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("n", [8, 1000, 4096 * 33 + 8, 1 << 20])
@pytest.mark.parametrize("src,dst", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32),
                                     (torch.float32, torch.bfloat16), (torch.int64, torch.int64)])
def test_gather_emulated_ranks(ext, world, n, src, dst):
    g = torch.Generator(device="cuda").manual_seed(n + world)
    if src == torch.int64:
        shards = [torch.randint(-2**40, 2**40, (n,), device="cuda", generator=g) for _ in range(world)]
    else:
        shards = [torch.randn(n, device="cuda", generator=g).to(src) for _ in range(world)]
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    for me in range(world):
        out = torch.empty(world, n, dtype=dst, device="cuda")
        ext.gather(out, _table(shards), n, src, me, True, status)
        want = torch.stack(shards).to(dst)
        assert torch.equal(out, want)
    assert int(status[0]) == 0


def test_gather_unaligned_rows(ext):
    world, n = 3, 1001  # 2002-byte rows: not a multiple of 16
    shards = [torch.randn(n, device="cuda").bfloat16() for _ in range(world)]
    out = torch.empty(world, n, dtype=torch.bfloat16, device="cuda")
    ext.gather(out, _table(shards), n, torch.bfloat16, 1, False, torch.zeros(4, dtype=torch.int32, device="cuda"))
    assert torch.equal(out, torch.stack(shards))


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("n", [4, 1000, 4096 * 9 + 4, 1 << 19, 1001])
@pytest.mark.parametrize("in_dtype,acc_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                                (torch.bfloat16, torch.bfloat16)])
def test_scatter_accumulate_emulated_ranks(ext, world, n, in_dtype, acc_dtype):
    """Every emulated rank adds its [world, n] rows into the owners; sums are exactly representable."""
    if n % 2 and acc_dtype == torch.bfloat16 and world > 1:
        pytest.skip("odd bf16 rows use the scalar path tested with world 1")
    g = torch.Generator(device="cuda").manual_seed(7)
    accs = [torch.zeros(n, dtype=acc_dtype, device="cuda") for _ in range(world)]
    ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    inputs = [torch.randint(-4, 5, (world, n), device="cuda", generator=g).to(in_dtype) for _ in range(world)]
    for rounds in range(2):
        for me in range(world):
            ext.scatter_accumulate(inputs[me], _table(accs), _table(ctrs), n, acc_dtype, me, 1.0, True, status)
    want = 2 * torch.stack(inputs).float().sum(0)  # [world, n]: row p belongs to owner p
    for p in range(world):
        assert torch.equal(accs[p].float(), want[p]), (p, (accs[p].float() - want[p]).abs().max())
        assert int(ctrs[p][0]) == 2 * world
    # the arrival wait succeeds at the dispatched count ...
    ext.wait_counter(ctrs[0], 2 * world, 1000, status)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    # ... and a count that nothing will ever deliver runs out of budget and reports, instead of hanging
    ext.wait_counter(ctrs[0], 2 * world + 1, 50, status)
    torch.cuda.synchronize()
    assert status[:3].tolist() == [1, 0, 2 * world]
    from odc_b200.runtime.status import OdcTimeoutError, check_status_word
    with pytest.raises(OdcTimeoutError):
        check_status_word(*status[:3].tolist())


def test_scatter_accumulate_scale(ext):
    n, world = 4096, 4
    accs = [torch.zeros(n, device="cuda") for _ in range(world)]
    ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
    x = torch.randint(-8, 8, (world, n), device="cuda").float()
    ext.scatter_accumulate(x, _table(accs), _table(ctrs), n, torch.float32, 0, 0.25, False,
                           torch.zeros(4, dtype=torch.int32, device="cuda"))
    assert torch.equal(torch.stack(accs), x * 0.25)


def test_scatter_accumulate_scale_on_the_device(ext):
    """A factor the host has not seen, on top of the one it passes; both input types (exact: powers of two)."""
    n, world = 4100, 3
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    for dtype in (torch.float32, torch.bfloat16):
        accs = [torch.ones(n, device="cuda") for _ in range(world)]
        ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
        x = torch.randint(-8, 8, (world, n), device="cuda").to(dtype)
        factor = torch.tensor(0.5, device="cuda")
        ext.scatter_accumulate(x, _table(accs), _table(ctrs), n, torch.float32, 1, 0.25, True, status, n, factor)
        assert torch.equal(torch.stack(accs), 1 + x.float() * 0.125)
        assert [int(c[0]) for c in ctrs] == [1] * world
    assert int(status[0]) == 0


@pytest.mark.parametrize("world,tokens,width,vocab", [(1, 1, 8, 4), (1, 700, 264, 50), (3, 700, 64, 100), (8, 3000, 2048, 1001)])
def test_embedding_scatter_emulated_ranks(ext, world, tokens, width, vocab):
    """Rows of the lookup's gradient in the owners' accumulators: repeated ids, the first and the last row, ids outside of the
    vocabulary skipped, padding rows untouched.  Whole numbers: exact in any order."""
    rows = -(-vocab // world)
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    ids = torch.randint(0, vocab, (tokens,), device="cuda", generator=gen)
    ids[: tokens // 3] = vocab - 1
    if tokens > 3:
        ids[-3:] = torch.tensor([0, -1, vocab], device="cuda")
    dx = torch.randint(-4, 5, (tokens, width), device="cuda", generator=gen).bfloat16()
    accs = [torch.ones(rows, width, device="cuda") for _ in range(world)]
    ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
    for _ in range(2):
        ext.embedding_scatter(ids, dx, _table(accs), _table(ctrs), rows, vocab, 0.5)
    want = torch.ones(world * rows, width, device="cuda", dtype=torch.float64)
    keep = (ids >= 0) & (ids < vocab)
    want.index_add_(0, ids[keep], dx[keep].double())
    assert torch.equal(torch.cat(accs).double(), want)
    assert [int(c[0]) for c in ctrs] == [2] * world


def test_post_and_wait_runs_out(ext):
    """The one launch of a synchronisation: posts and waits; a producer that never posts, and fewer arrivals than announced,
    run into the short limit and are named, and the context stays usable."""
    nprod = 3
    slots, ctr = (torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(2))
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    host = torch.zeros(4, dtype=torch.int32).pin_memory()
    addrs = [slots.data_ptr() + 8 * p for p in range(nprod)]
    ctr[0] = 6
    assert ext.post_and_wait(addrs, [1, 2, 3], 1, slots, nprod, ctr, 500, status, host) == (0, 0, 0)
    assert [int(v) >> 32 for v in slots[:nprod]] == [1] * nprod
    assert ext.post_and_wait(addrs[:2], [1, 2], 2, slots, nprod, ctr, 50, status, host) == (1, 1000 + nprod - 1, 1)
    status.zero_()
    assert ext.post_and_wait(addrs, [1, 2, 4], 3, slots, nprod, ctr, 50, status, host) == (1, 0, 6)
    status.zero_()
    ctr[0] = 7
    assert ext.post_and_wait(addrs, [1, 2, 4], 4, slots, nprod, ctr, 500, status, host) == (0, 0, 0)


# ------------------------------------------------------------------------------------ elementwise
@pytest.mark.parametrize("rows,cols", [(1, 256), (333, 2048), (4096, 5120), (17, 8192)])
def test_rmsnorm(rows, cols):
    from odc_b200 import ops
    from odc_b200.ops import reference as ref
    x = torch.randn(rows, cols, device="cuda").bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(cols, device="cuda")).bfloat16().requires_grad_()
    y = ops.rms_norm(x, w, 1e-5)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yr = ref.rms_norm(xr, wr, 1e-5)
    yr.backward(dy.float())
    torch.testing.assert_close(y.float(), yr, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, rtol=2e-2, atol=2e-2 * math.sqrt(rows))


@pytest.mark.parametrize("nq,nkv,d", [(4, 4, 64), (32, 8, 64), (40, 8, 128)])
def test_rope(nq, nkv, d):
    from odc_b200 import ops
    from odc_b200.ops import reference as ref
    T = 257
    qkv = torch.randn(T, (nq + 2 * nkv) * d, device="cuda").bfloat16().requires_grad_()
    pos = torch.randint(0, 30000, (T,), device="cuda")
    out = ops.rope_qkv(qkv, pos, nq, nkv, d, 500000.0)
    dout = torch.randn_like(out)
    out.backward(dout)
    x = qkv.detach().float().cpu().requires_grad_()
    q, k, v = x.split([nq * d, nkv * d, nkv * d], dim=-1)
    want = torch.cat([ref.rope(q.reshape(T, nq, d), pos.cpu(), 500000.0).reshape(T, -1),
                      ref.rope(k.reshape(T, nkv, d), pos.cpu(), 500000.0).reshape(T, -1), v], dim=-1)
    want.backward(dout.float().cpu())
    torch.testing.assert_close(out.float().cpu(), want, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(qkv.grad.float().cpu(), x.grad, rtol=2e-2, atol=2e-2)


def test_swiglu():
    from odc_b200 import ops
    from odc_b200.ops import reference as ref
    gu = torch.randn(513, 2 * 1376, device="cuda").bfloat16().requires_grad_()
    y = ops.swiglu(gu)
    dy = torch.randn_like(y)
    y.backward(dy)
    g = gu.detach().float().requires_grad_()
    yr = ref.swiglu(g)
    yr.backward(dy.float())
    torch.testing.assert_close(y.float(), yr, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(gu.grad.float(), g.grad, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("T,V", [(100, 1024), (300, 128256)])
def test_ce_fwd_bwd(ext, T, V):
    logits = (3 * torch.randn(T, V, device="cuda")).bfloat16()
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[5] = -100
    scale = torch.rand(T, device="cuda")
    lf = logits.float().requires_grad_()
    keep = labels != -100
    want = (torch.nn.functional.cross_entropy(lf, labels, reduction="none", ignore_index=-100) * scale).sum()
    want.backward()
    loss = torch.zeros((), device="cuda")
    ext.ce_fwd_bwd(logits, labels, scale, loss, -100)
    torch.testing.assert_close(loss, want.detach(), rtol=1e-3, atol=1e-3)
    torch.testing.assert_close(logits.float(), lf.grad, rtol=2e-2, atol=1e-4)
    assert float(logits[~keep].abs().sum()) == 0.0


def test_token_logprobs_kernel_reads_only(ext):
    """Forward-only instantiation of the cross-entropy kernel: per-row log-probability of the label, 0 for ignored
    rows, logits left untouched."""
    T, V = 300, 1000
    logits = (3 * torch.randn(T, V, device="cuda")).bfloat16()
    keep = logits.clone()
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[::7] = -100
    out = torch.full((T,), 7.0, device="cuda")
    ext.token_logprobs(logits, labels, out, -100)
    want = logits.float().log_softmax(-1).gather(-1, labels.clamp_min(0)[:, None]).squeeze(-1)
    want = torch.where(labels != -100, want, torch.zeros_like(want))
    torch.testing.assert_close(out, want, rtol=1e-4, atol=2e-4)
    assert torch.equal(logits, keep)


def test_adamw_matches_torch(ext):
    n = 100003
    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda")
    ref_p = torch.nn.Parameter(p.clone())
    opt = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    m, v, low = torch.zeros_like(p), torch.zeros_like(p), torch.empty(n, dtype=torch.bfloat16, device="cuda")
    for step in range(1, 4):
        ref_p.grad = g * step
        opt.step()
        ext.adamw_step(p, g * step, m, v, low, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, 1.0)
    torch.testing.assert_close(p, ref_p.detach(), rtol=1e-5, atol=1e-6)
    assert torch.equal(low, p.bfloat16())


@pytest.mark.parametrize("grad", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,skip", [(1, 0), (3, 0), (4, 0), (1025, 0), (4098, 1), (4098, 4)])
def test_adamw_accesses(ext, n, skip, grad):
    """Wide and element-wise accesses, remainders, arrays that start off a 16-byte boundary: the same numbers."""
    base = [torch.rand(n + skip, device="cuda") for _ in range(3)]
    g = torch.randn(n + skip, device="cuda").to(grad)[skip:]
    p, m, v = (t[skip:] for t in base)
    low = torch.zeros(n + skip, dtype=torch.bfloat16, device="cuda")[skip:]
    pd, md, vd, gd = p.double(), m.double(), v.double(), g.double() * 0.5
    ext.adamw_step(p, g, m, v, low, 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, 0.5)
    md, vd = 0.9 * md + 0.1 * gd, 0.95 * vd + 0.05 * gd * gd
    pd = pd * (1 - 1e-3) - 1e-2 / (1 - 0.9 ** 3) * md / (vd.sqrt() / (1 - 0.95 ** 3) ** 0.5 + 1e-8)
    for got, exp in ((p, pd), (m, md), (v, vd)):
        torch.testing.assert_close(got.double(), exp, rtol=2e-5, atol=2e-6)
    assert torch.equal(low, p.bfloat16())


@pytest.mark.parametrize("n,skip", [(4096, 0), (4097, 0), (4099, 0), (4097, 1)])
def test_adamw_is_one_launch(ext, n, skip):
    """A remainder of four has no launch of its own (2 us, a fifth of the update of two million elements)."""
    p, m, v, g = (torch.rand(n + skip, device="cuda")[skip:] for _ in range(4))
    ext.adamw_step(p, g, m, v, None, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1, 1.0)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        ext.adamw_step(p, g, m, v, None, 1e-2, 0.9, 0.95, 1e-8, 0.1, 2, 1.0)
        torch.cuda.synchronize()
    assert sum("adamw" in e.name for e in prof.events()) == 1


# ------------------------------------------------------------------------------------ GEMM
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (300, 1376, 200), (1000, 264, 1032),
                                   (4096, 2048, 4096)])
def test_gemm_layouts(ext, layout, M, N, K):
    K = (K + 7) // 8 * 8 if layout != "tn" else K
    M = (M + 7) // 8 * 8 if layout == "tn" else M
    torch.manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda").bfloat16()
    B = torch.randn(K, N, device="cuda").bfloat16()
    want = A.float() @ B.float()
    a = A.t().contiguous() if layout == "tn" else A
    b = B.t().contiguous() if layout == "nt" else B
    c = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ext.gemm(a, b, c, layout, None, False)
    torch.cuda.synchronize()
    assert ext.kernel_status()[0].item() == 0
    torch.testing.assert_close(c.float(), want, rtol=2e-2, atol=2e-2 * math.sqrt(K))
    # fp32 output with accumulation and bias
    bias = torch.randn(N, device="cuda").bfloat16()
    c32 = torch.ones(M, N, device="cuda")
    ext.gemm(a, b, c32, layout, bias, True)
    torch.testing.assert_close(c32, want + 1 + bias.float(), rtol=1e-2, atol=1e-2 * math.sqrt(K))


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (256, 512, 256), (304, 1376, 200), (1000, 264, 1032),
                                   (4096, 2048, 4096), (16384, 3072, 2048)])
def test_gemm_cta_pair_layouts(ext, layout, M, N, K):
    """The CTA-pair (cta_group::2) kernel, forced: 256 x 256 tiles split over two SMs, ragged edges in M, N and K."""
    K = (K + 7) // 8 * 8 if layout != "tn" else K
    M = (M + 7) // 8 * 8 if layout == "tn" else M
    torch.manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda").bfloat16()
    B = torch.randn(K, N, device="cuda").bfloat16()
    want = A.float() @ B.float()
    a = A.t().contiguous() if layout == "tn" else A
    b = B.t().contiguous() if layout == "nt" else B
    c = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ext.gemm(a, b, c, layout, None, False, None, 1)
    torch.cuda.synchronize()
    assert ext.kernel_status()[0].item() == 0, ext.kernel_status().tolist()
    torch.testing.assert_close(c.float(), want, rtol=2e-2, atol=2e-2 * math.sqrt(K))
    # bias + residual in the epilogue of a bf16 output
    bias = torch.randn(N, device="cuda").bfloat16()
    res = torch.randn(M, N, device="cuda").bfloat16()
    ext.gemm(a, b, c, layout, bias, False, res, 1)
    torch.testing.assert_close(c.float(), want + bias.float() + res.float(), rtol=2e-2, atol=2e-2 * math.sqrt(K))
    # fp32 output with accumulation (TMA reduce-add) and bias
    c32 = torch.ones(M, N, device="cuda")
    ext.gemm(a, b, c32, layout, bias, True, None, 1)
    torch.cuda.synchronize()
    assert ext.kernel_status()[0].item() == 0, ext.kernel_status().tolist()
    torch.testing.assert_close(c32, want + 1 + bias.float(), rtol=1e-2, atol=1e-2 * math.sqrt(K))
    # fp32 output, plain store over whatever the buffer held
    c32.fill_(float("nan"))
    ext.gemm(a, b, c32, layout, None, False, None, 1)
    torch.testing.assert_close(c32, want, rtol=1e-2, atol=1e-2 * math.sqrt(K))


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K", [(512, 4736, 72), (512, 4744, 72), (264, 376, 136), (256, 264, 64), (776, 392, 1600)])
def test_gemm_tiles_of_half_the_width(ext, layout, M, N, K):
    """37 x 2 tiles of 256 x 128 have a pair each and are taken, 38 x 2 would take two rounds; edges in the last half tile.  Against 64 bits, with
    bias and residual: fp32 sums (2e-6 of the magnitudes) and one rounding to bf16."""
    for a, b, c, lay, _, _, want, bound in _group_case([(layout, M, N, K, torch.bfloat16, False, 1.0)]):
        bias, res = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16()
        ext.gemm(a, b, c, lay, None, False, None, 1)
        assert ((c.double() - want).abs() <= bound).all()
        full = want + bias.double() + res.double()
        ext.gemm(a, b, c, lay, bias, False, res, 1)
        assert ((c.double() - full).abs() <= bound + 2e-6 * (bias.double().abs() + res.double().abs()) + full.abs() * 2.0 ** -8).all()


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K,divided", [(8, 256, 4096, True), (136, 1536, 8968, True), (255, 2048, 2048, False),
                                           (256, 256, 2048, True), (264, 264, 4040, True), (765, 1536, 17920, True),
                                           (520, 1544, 8968, True), (768, 2048, 1536, False), (2304, 2304, 4096, False)])
def test_gemm_divided_reduction(ext, layout, M, N, K, divided):
    """Few tiles and a long reduction: partial products and their sum, ragged tiles and a ragged last part included."""
    M = (M + 7) // 8 * 8 if layout == "tn" else M
    assert (ext.gemm_split_bytes(M, N, K) > 0) == divided
    torch.manual_seed(M + N + K)
    A, B = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    bias, res = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N + 8, device="cuda").bfloat16()[:, :N]
    a = A.t().contiguous() if layout == "tn" else A
    b = B.t().contiguous() if layout == "nt" else B
    want = A.double() @ B.double()
    c = torch.empty(M, N + 16, dtype=torch.bfloat16, device="cuda")[:, :N]
    for kw, exp in (((None, False), want), ((bias, False, res), want + bias.double() + res.double())):
        ext.gemm(a, b, c, layout, *kw)
        torch.cuda.synchronize()
        assert ext.kernel_status()[0].item() == 0, ext.kernel_status().tolist()
        # fp32 sums of K products (sqrt(K) 2^-24 each way, far below) and one rounding to bf16
        assert ((c.double() - exp).abs() <= 2 ** -8 * exp.abs() + 1e-4 * K ** 0.5).all()


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K", [(3072, 2048, 8200), (2996, 2056, 8200), (5000, 1800, 8192)])
def test_gemm_divided_last_round(ext, layout, M, N, K):
    """A few tiles more than the pairs can take in whole rounds: only those are divided, the others stored as they are."""
    M = (M + 7) // 8 * 8 if layout == "tn" else M
    torch.manual_seed(M + N + K)
    A, B = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    bias, res = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N + 8, device="cuda").bfloat16()[:, :N]
    a = A.t().contiguous() if layout == "tn" else A
    b = B.t().contiguous() if layout == "nt" else B
    want = A.double() @ B.double()
    tiles, whole, parts, scratch = ext.gemm_plan(M, N, K, torch.cuda.get_device_properties(0).multi_processor_count)
    assert 0 < whole < tiles and parts > 1 and ext.gemm_split_bytes(M, N, K) == 0
    c = torch.empty(M, N + 16, dtype=torch.bfloat16, device="cuda")[:, :N]
    for kw, exp in (((None, False), want), ((bias, False, res), want + bias.double() + res.double())):
        before, held = ext.kernel_launches(), torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        ext.gemm(a, b, c, layout, *kw)
        torch.cuda.synchronize()
        assert ext.kernel_launches() - before == 1   # the sum of the parts
        assert scratch <= torch.cuda.max_memory_allocated() - held < scratch + (2 << 20)
        assert ext.kernel_status()[0].item() == 0, ext.kernel_status().tolist()
        # fp32 sums of K products (sqrt(K) 2^-24 each way, far below) and one rounding to bf16
        assert ((c.double() - exp).abs() <= 2 ** -8 * exp.abs() + 1e-4 * K ** 0.5).all()


@pytest.mark.parametrize("T,n_out,k_in", [(1900, 512, 512), (1900, 768, 520), (4099, 3072, 2048)])
def test_wgrad_scatter_divided(ext, T, n_out, k_in):
    """Few tiles, or a last round of few: their parts meet in the accumulator; under deterministic algorithms none does."""
    torch.manual_seed(T + n_out)
    dy, x = torch.randn(T, n_out, device="cuda").bfloat16(), torch.randn(T, k_in, device="cuda").bfloat16()
    rows = (n_out + 127) // 128 * 128
    ctr = torch.zeros(8, dtype=torch.int64, device="cuda")

    def run():
        acc = torch.ones(rows, k_in, device="cuda")
        assert ext.gemm_wgrad_scatter_tma(dy, x, [acc.data_ptr()], _table([ctr]), 0, rows, 0.5, 0)
        torch.cuda.synchronize()
        assert ext.kernel_status()[0].item() == 0
        return acc

    want = 1 + 0.5 * (dy.double().t() @ x.double())
    # fp32 sums of T products of unit size: a few 2^-24 sqrt(T) of their magnitude sqrt(T), whatever the order
    bound = 2 ** -20 * T
    assert (run()[:n_out].double() - want).abs().max().item() < bound
    torch.use_deterministic_algorithms(True)
    try:
        first = run()
        assert (first[:n_out].double() - want).abs().max().item() < bound
        assert all(torch.equal(first, run()) for _ in range(3))
    finally:
        torch.use_deterministic_algorithms(False)
    assert int(ctr[0]) == 5


def _group_case(products, seed=0):
    """Operands of (layout, M, N, K, output, added) each, row strides wider than the rows, and the result in 64 bits."""
    torch.manual_seed(seed)
    out = []
    for lay, M, N, K, dtype, add, scale in products:
        wide = lambda r, c: torch.randn(r, c + 8, device="cuda").bfloat16()[:, :c]
        a, b = wide(*((K, M) if lay == "tn" else (M, K))), wide(*((N, K) if lay == "nt" else (K, N)))
        c = torch.randn(M, N + 8, device="cuda").to(dtype)[:, :N]
        A, B = (a.t() if lay == "tn" else a).double(), (b.t() if lay == "nt" else b).double()
        want = (A @ B) * scale + (c.double() if add else 0)
        # fp32 sums of K products: a few units in the last place of the sum of magnitudes; then one rounding to the output's type
        bound = (A.abs() @ B.abs() * scale + c.double().abs()) * 2e-6 + want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23)
        out.append((a, b, c, lay, add, scale, want, bound))
    return out


@pytest.mark.parametrize("parts,products", [
    # (layout, M, N, K, output, added, scale); bf16 tiles in up to eight parts, edges in M, N and K, one to three products
    ([1, 1], [("nn", 8, 256, 64, torch.bfloat16, False, 1.0), ("tn", 264, 520, 72, torch.bfloat16, False, 1.0)]),
    (None, [("nn", 300, 264, 8200, torch.bfloat16, False, 1.0), ("tn", 776, 264, 300, torch.float32, False, 0.5)]),
    (None, [("nn", 257, 512, 32768, torch.bfloat16, False, 1.0), ("tn", 256, 256, 257, torch.bfloat16, False, 1.0),
            ("nt", 255, 264, 200, torch.float32, False, 2.0)]),
    (None, [("tn", 512, 512, 4104, torch.float32, True, 0.25), ("tn", 1536, 264, 4104, torch.float32, True, 1.0)]),
    (None, [("nn", 1000, 1536, 4096, torch.bfloat16, False, 1.0), ("tn", 4096, 1536, 1000, torch.float32, True, 1.0),
            ("tn", 1536, 2048, 1000, torch.bfloat16, False, 1.0)]),
    (None, [("nn", 64, 256, 5000, torch.bfloat16, False, 1.0)]),
    # tiles of half the width next to whole ones
    ([1, 1], [("nn", 300, 392, 2048, torch.bfloat16, False, 1.0), ("tn", 2048, 392, 304, torch.float32, True, 1.0)]),
    (None, [("nt", 300, 1160, 1024, torch.float32, False, 1.0), ("nn", 264, 264, 512, torch.bfloat16, False, 1.0)]),
])
def test_groups_of_products(ext, parts, products):
    ops = _group_case(products)
    plan = ext.gemm_group_plan([(M, N, K, d == torch.float32, add) for _, M, N, K, d, add, _ in products], ext.sm_count())
    assert all(1 <= s <= 8 for s in plan) and (parts is None or plan == parts)
    start = [c.clone() for _, _, c, *_ in ops]
    for _ in range(3):   # the counters of one launch are as the next one expects them
        for (_, _, c, *_), c0 in zip(ops, start):
            c.copy_(c0)
        assert ext.gemm_group([(a, b, c, lay, add, scale) for a, b, c, lay, add, scale, _, _ in ops])
        for a, b, c, lay, add, scale, want, bound in ops:
            assert ((c.double() - want).abs() <= bound).all(), (lay, plan)


@pytest.mark.parametrize("products", [
    # all tiles in parts, those of the last round, none; ragged edges; next to products of other kinds
    [("nn", 765, 1536, 17920), ("tn", 17920, 1536, 765), ("tn", 1536, 8960, 765)],
    [("nn", 4090, 1544, 20000), ("tn", 1024, 1544, 4090)],
    [("tn", 3072, 2056, 16400), ("nn", 2304, 2304, 16400), ("nt", 1000, 264, 17000)],
    [("nn", 2304, 2304, 16400)], [("tn", 264, 264, 17000)], [("nn", 600, 520, 200), ("tn", 520, 200 * 8, 600)]])
def test_groups_give_the_bytes_of_single_products(ext, products):
    """A bf16 result does not depend on what is formed in the same launch: a sum over more than 16384 is divided as in a launch of its own."""
    ops = [case[:4] for case in _group_case([(lay, M, N, K, torch.bfloat16, False, 1.0) for lay, M, N, K in products])]
    assert ext.gemm_group([(a, b, c, lay, False, 1.0) for a, b, c, lay in ops])
    for a, b, c, lay in ops:
        alone = torch.empty_like(c)
        ext.gemm(a, b, alone, lay, None, False)
        assert torch.equal(c, alone), (lay, *c.shape)


def test_parts_of_a_group_are_summed_in_one_order(ext):
    """Eight parts and as many CTAs that may come last: the same bytes every time, in a replayed graph as well."""
    torch.manual_seed(0)
    a, b = torch.randn(300, 30000, device="cuda").bfloat16(), torch.randn(30000, 512, device="cuda").bfloat16()
    x = torch.randn(300, 264, device="cuda").bfloat16()
    outs = [torch.empty(300, 512, device="cuda", dtype=torch.bfloat16) for _ in range(6)]
    dw = torch.empty(30000, 264, device="cuda", dtype=torch.bfloat16)
    run = lambda o: ext.gemm_group([(a, b, o, "nn", False, 1.0), (a, x, dw, "tn", False, 1.0)])
    for o in outs[:3]:
        assert run(o)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        for o in outs[3:]:
            run(o)
    for _ in range(3):
        for o in outs[3:]:
            o.zero_()
        g.replay()
        assert all(torch.equal(o, outs[0]) for o in outs)
    assert ext.gemm_group_plan([(300, 512, 30000, False, False), (30000, 264, 300, False, False)], ext.sm_count())[0] > 1


def test_groups_that_are_not_taken(ext):
    """Types, widths and alignments the kernel does not read or write: nothing is done, the products go one by one."""
    t = lambda *s, dtype=torch.bfloat16: torch.zeros(*s, device="cuda", dtype=dtype)
    good = (t(300, 512), t(512, 256), t(300, 256), "nn", False, 1.0)
    for bad in ((t(300, 512).float(), t(512, 256).float(), t(300, 256).float(), "nn", False, 1.0),
                (t(300, 512), t(512, 200), t(300, 200), "nn", False, 1.0), (t(300, 512), t(512, 260), t(300, 260), "nn", False, 1.0),
                (t(300, 32), t(32, 256), t(300, 256), "nn", False, 1.0), (t(300, 512), t(512, 256), t(300, 256), "nn", True, 1.0),
                (t(300, 516)[:, 4:], t(512, 256), t(300, 256), "nn", False, 1.0)):
        assert not ext.gemm_group([good, bad])
    assert not ext.gemm_group([good] * 4)


@pytest.mark.parametrize("T,H,F", [(24, 256, 512), (300, 512, 1536), (765, 1536, 8960)])
def test_chained_kernels_see_their_predecessors(ext, T, H, F):
    """A kernel may start before the one ahead of it has ended: a chain queued without a pause gives the bytes of one that is
    waited for after every call, also when each link reuses the memory of the link before."""
    torch.manual_seed(T)
    x0 = torch.randn(T, H, device="cuda").bfloat16()
    w = torch.rand(H, device="cuda").bfloat16()
    up, down = (0.05 * torch.randn(n, k, device="cuda").bfloat16() for n, k in ((2 * F, H), (H, F)))

    def chain(pause):
        x = x0
        for _ in range(6):
            for step in (lambda t: ext.rmsnorm_fwd(t, w, 1e-5)[0], lambda t: ext.linear(t, up), ext.swiglu_fwd,
                         lambda t: ext.linear(t, down)):
                x = step(x)
                if pause:
                    torch.cuda.synchronize()
        return x

    want = chain(True)
    assert torch.isfinite(want.float()).all()
    for _ in range(5):
        assert torch.equal(chain(False), want)


def _same_bytes_without_pauses(steps, tries=5):
    """``steps``: functions of the value before; a run that waits after each, then runs that do not."""
    def run(pause):
        x = None
        for step in steps:
            x = step(x)
            if pause:
                torch.cuda.synchronize()
        return x
    want = [t.clone() for t in run(True)]
    assert all(torch.isfinite(t.float()).all() for t in want)
    for _ in range(tries):
        for got, exp in zip(run(False), want):
            assert torch.equal(got, exp)


@pytest.mark.parametrize("T,H,V", [(8, 256, 1024), (300, 512, 32000)])
def test_chained_softmax_kernels_see_their_predecessors(ext, T, H, V):
    """Product -> log-probabilities, product -> gradient of the logits -> product, in one logits buffer."""
    torch.manual_seed(T)
    hs = [torch.randn(T, H, device="cuda").bfloat16() for _ in range(4)]
    w = (torch.randn(V, H, device="cuda") / 16).bfloat16()
    ids, scale = torch.randint(0, V, (T,), device="cuda"), torch.rand(T, device="cuda")
    logits = torch.empty(T, V, device="cuda", dtype=torch.bfloat16)
    lp = torch.empty(len(hs), T, device="cuda")
    dh = torch.empty(len(hs), T, H, device="cuda", dtype=torch.bfloat16)
    loss = torch.zeros((), device="cuda")
    steps = []
    for i, h in enumerate(hs):
        steps += [lambda _, h=h: ext.gemm(h, w, logits, "nt", None, False),
                  lambda _, i=i: ext.token_logprobs(logits, ids, lp[i], -100),
                  lambda _, h=h: ext.gemm(h, w, logits, "nt", None, False),
                  lambda _: ext.ce_fwd_bwd(logits, ids, scale, loss, -100),
                  lambda _, i=i: ext.gemm(logits, w, dh[i], "nn", None, False)]
    _same_bytes_without_pauses(steps + [lambda _: (lp, dh)])


@pytest.mark.parametrize("d", [64, 128])
def test_chained_attention_kernels_see_their_predecessors(ext, d):
    """Rotation -> attention forward -> backward with reused memory; sequences of one key tile, whose gradients are sums in a
    fixed order."""
    lens, hq, hkv = [100, 128, 37], 4, 2
    T = sum(lens)
    torch.manual_seed(d)
    qkvs = [torch.randn(T, (hq + 2 * hkv) * d, device="cuda").bfloat16() for _ in range(4)]
    do = torch.randn(T, hq, d, device="cuda").bfloat16()
    pos = torch.cat([torch.arange(n) for n in lens]).cuda()
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).int()
    out = torch.empty(len(qkvs), T, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16)

    def split(x):
        return tuple(t.view(T, -1, d) for t in x.split([hq * d, hkv * d, hkv * d], dim=-1))

    steps = []
    for i, qkv in enumerate(qkvs):
        steps += [lambda _, qkv=qkv: ext.rope_qkv(qkv, pos, hq, hkv, d, 10000.0, False),
                  lambda x: (x, *ext.attn_fwd(*split(x), cu, max(lens), True, d ** -0.5)),
                  lambda x: ext.attn_bwd(do, *split(x[0]), x[1], x[2], cu, max(lens), True, d ** -0.5, True)[3],
                  lambda g: ext.rope_qkv(g, pos, hq, hkv, d, 10000.0, True),
                  lambda g, i=i: out[i].copy_(g)]
    _same_bytes_without_pauses(steps + [lambda _: (out,)])


_WITHOUT_PAIRS = """
import torch
from odc_b200 import ops, _ext
ext = _ext.load()
a, b = torch.randn(765, 17920, device="cuda").bfloat16(), torch.randn(1536, 17920, device="cuda").bfloat16()
assert ext.gemm_split_bytes(765, 1536, 17920) > 0
out = torch.empty(765, 1536, device="cuda", dtype=torch.bfloat16)
ops.gemm(a, b, out=out)
torch.cuda.synchronize()
torch.cuda.reset_peak_memory_stats()
before, held = ops.kernel_launches(), torch.cuda.memory_allocated()
ops.gemm(a, b, out=out)
assert ops.kernel_launches() - before == 1, ops.kernel_launches() - before
assert torch.cuda.max_memory_allocated() == held, (torch.cuda.max_memory_allocated(), held)
"""


def test_single_cta_products_allocate_and_count_nothing_for_a_division():
    """ODC_GEMM_PAIR=0 is read once per process: a process of its own."""
    import subprocess
    import sys
    r = subprocess.run([sys.executable, "-c", _WITHOUT_PAIRS], env={**os.environ, "ODC_GEMM_PAIR": "0"}, capture_output=True,
                       text=True, timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr


def _linear(x, w, b):
    from odc_b200 import ops
    with torch.no_grad():
        return ops.linear(x, w, b)


@pytest.mark.parametrize("T,H,nq,nkv,d,bias", [(256, 64, 2, 1, 64, False), (300, 264, 5, 1, 64, True), (1000, 512, 8, 2, 64, False),
                                               (256, 128, 1, 1, 128, True), (520, 200, 12, 2, 128, True), (16, 128, 4, 4, 64, True),
                                               (300, 8960, 4, 1, 128, False), (2600, 2048, 32, 8, 64, False), (560, 5120, 40, 8, 128, True)])
def test_projection_with_rotation(ext, T, H, nq, nkv, d, bias):
    """The bytes of the product and the pass over it.  Fewer rows than a tile and products divided as a whole or in their last round take
    those."""
    torch.manual_seed(0)
    x, w = torch.randn(T, H, device="cuda").bfloat16(), (torch.randn((nq + 2 * nkv) * d, H, device="cuda") * H ** -0.5).bfloat16()
    b = torch.randn(w.shape[0], device="cuda").bfloat16() if bias else None
    pos = torch.arange(T, device="cuda") % 777 * 3
    out = ext.linear_rope(x, w, b, pos, nq, nkv, d, 10000.0)
    assert torch.equal(out, ext.rope_qkv(_linear(x, w, b), pos, nq, nkv, d, 10000.0, False))


@pytest.mark.parametrize("M,N,K", [(300, 264, 128), (1000, 520, 256), (1000, 512, 128), (765, 1536, 8960), (2304, 2304, 4096), (16, 264, 128)])
@pytest.mark.parametrize("offset", [1, 4])
def test_bias_that_starts_off_a_16_byte_boundary(ext, M, N, K, offset):
    """A view of a larger vector, in bf16 and fp32 results, with a residual, in half-width, divided and single-CTA products, gathered
    weights and the rotary projection: the bytes that the same bias gives at the start of an allocation."""
    torch.manual_seed(0)
    x, w = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    bias, res = torch.randn(N + 8, device="cuda").bfloat16()[offset:offset + N], torch.randn(M, N, device="cuda").bfloat16()
    whole = bias.clone()
    assert bias.data_ptr() % 16 and whole.data_ptr() % 16 == 0

    def results(b):
        c, c32 = torch.empty_like(res), torch.ones(M, N, device="cuda")
        ext.gemm(x, w, c, "nt", b, False, res)
        ext.gemm(x, w, c32, "nt", b, True)
        out = [_linear(x, w, b), c, c32]
        if M >= 256:
            out.append(ext.gemm_gather(x, _table([w]), torch.empty_like(w), b, N, 0, res))
        if N == 512:
            out.append(ext.linear_rope(x, w, b, torch.arange(M, device="cuda"), N // 64 - 4, 2, 64, 10000.0))
        return out
    for got, want in zip(results(bias), results(whole)):
        assert torch.equal(got, want)
    assert ext.kernel_status()[0].item() == 0, ext.kernel_status().tolist()


def test_positions_that_are_a_strided_view(ext):
    """Every second value of a larger vector: what the same values give next to one another, in the op, its backward and a layer."""
    from odc_b200 import ops
    from odc_b200.models import DecoderLayer, get_config
    torch.manual_seed(0)
    with torch.device("cuda"):
        layer = DecoderLayer(get_config("tiny")).bfloat16()
    with torch.no_grad():
        for p in layer.parameters():
            p.normal_(0.0 if p.dim() == 2 else 1.0, 0.05)
    x = torch.randn(300, 256, device="cuda").bfloat16()
    cu = torch.tensor([0, 300], dtype=torch.int32, device="cuda")
    pos = torch.arange(600, device="cuda")[::2]
    qkv, dy = torch.randn(300, 768, device="cuda").bfloat16().requires_grad_(), torch.randn(300, 768, device="cuda").bfloat16()
    rotated = [ops.rope_qkv(qkv, p, 4, 4, 64, 10000.0) for p in (pos, pos.clone(memory_format=torch.contiguous_format))]
    assert not pos.is_contiguous() and torch.equal(*rotated)
    assert torch.equal(*(torch.autograd.grad(y, [qkv], dy)[0] for y in rotated))
    with torch.no_grad():
        assert torch.equal(layer(x, pos, cu, 300), layer(x, pos.contiguous(), cu, 300))


def test_positions_and_offsets_on_the_host_are_refused(ext):
    """A layer, its projection, rotation and attention name the device instead of handing a host address to a kernel."""
    from odc_b200 import ops
    from odc_b200.models import DecoderLayer, get_config
    with torch.device("cuda"):
        layer = DecoderLayer(get_config("tiny")).bfloat16()
    x = torch.randn(300, 256, device="cuda").bfloat16()
    pos, cu = torch.arange(300), torch.tensor([0, 300], dtype=torch.int32)
    qkv = torch.randn(300, 768, device="cuda").bfloat16()
    for call in (lambda: layer(x, pos, cu.cuda(), 300), lambda: layer(x, pos.cuda(), cu, 300), lambda: ops.rope_qkv(qkv, pos, 4, 4, 64, 10000.0),
                 lambda: ext.linear_rope(x, qkv.t()[:, :256].contiguous(), None, pos, 4, 4, 64, 10000.0), lambda: ops.varlen_attention_qkv(qkv, 4, 4, 64, cu, 300)):
        with pytest.raises(RuntimeError, match="on cpu"):
            call()


@pytest.mark.parametrize("T", [16, 300])
def test_projection_with_rotation_refuses_a_bias_of_another_length(ext, T):
    x, w = torch.randn(T, 128, device="cuda").bfloat16(), torch.randn(512, 128, device="cuda").bfloat16()
    for n in (8, 504, 520):
        with pytest.raises(RuntimeError, match="linear_rope: bias"):
            ext.linear_rope(x, w, torch.randn(n, device="cuda").bfloat16(), torch.arange(T, device="cuda"), 4, 2, 64, 10000.0)


@pytest.mark.parametrize("T,K,F", [(256, 128, 128), (300, 264, 1000), (520, 2048, 136), (1000, 512, 4160), (16, 128, 256),
                                   (765, 17920, 768)])
def test_linear_swiglu_matches_the_two_passes(ext, T, K, F):
    """Activation in the epilogue (ragged rows and columns of both halves) or, for few rows and divided reductions, behind it:
    the bytes of product and activation one after the other, forward and backward, with and without gradients."""
    torch.manual_seed(T + F)
    x = torch.randn(2, T // 2, K, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(2 * F, K, device="cuda") / K ** 0.5).bfloat16().requires_grad_()
    dy = torch.randn(2, T // 2, F, device="cuda").bfloat16()
    y = ext.linear_swiglu(x, w)
    want = ext.swiglu(ext.linear(x, w))
    with torch.no_grad():
        plain = ext.linear_swiglu(x, w)
    torch.cuda.synchronize()
    assert ext.kernel_status()[0].item() == 0, ext.kernel_status().tolist()
    assert torch.equal(y, want) and torch.equal(plain, want)
    for a, b in zip(torch.autograd.grad(y, [x, w], dy), torch.autograd.grad(want, [x, w], dy)):
        assert torch.equal(a, b)


def test_linear_autograd_matches_reference():
    from odc_b200 import ops
    x = torch.randn(3, 100, 512, device="cuda").bfloat16().requires_grad_()
    w = (0.05 * torch.randn(768, 512, device="cuda")).bfloat16().requires_grad_()
    b = torch.randn(768, device="cuda").bfloat16().requires_grad_()
    y = ops.linear(x, w, b)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_() for t in (x, w, b))
    yr = torch.nn.functional.linear(xr, wr, br)
    yr.backward(dy.float())
    torch.testing.assert_close(y.float(), yr, rtol=2e-2, atol=5e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=2e-2, atol=5e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, rtol=2e-2, atol=0.5)
    torch.testing.assert_close(b.grad.float(), br.grad, rtol=2e-2, atol=0.5)


@pytest.mark.parametrize("T,H,V", [(1, 64, 256), (63, 264, 1000), (300, 512, 4096), (700, 256, 32000), (1000, 1536, 8192)])
@pytest.mark.parametrize("factor", [1.0, 1 / 3])
def test_loss_of_one_chunk_keeps_the_logit_gradients(T, H, V, factor):
    """One chunk (the gradient of the logits waits for the backward) and several (the weight's gradient in fp32 does), both against
    64 bits: the same loss, and gradients no further from it."""
    from odc_b200 import ops
    torch.manual_seed(0)
    h, w = torch.randn(T, H, device="cuda").bfloat16(), (torch.randn(V, H, device="cuda") * H ** -0.5).bfloat16()
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[:: 7] = -100
    scale = torch.rand(T, device="cuda")
    hd, wd = h.double().requires_grad_(), w.double().requires_grad_()
    nll = torch.nn.functional.cross_entropy(hd @ wd.t(), labels, ignore_index=-100, reduction="none")
    want = torch.autograd.grad((nll * scale.double()).sum() * factor, [hd, wd])
    far = []
    for chunk in (T, max(1, T - 1)):
        a, b = h.clone().requires_grad_(), w.clone().requires_grad_()
        loss = ops.linear_cross_entropy(a, b, labels, scale, chunk=chunk)
        (loss * factor).backward()
        far.append([float((g.double() - x).norm() / x.norm()) if float(x.norm()) else float(g.double().norm()) for g, x in zip((a.grad, b.grad), want)])
        assert a.grad.dtype == b.grad.dtype == torch.bfloat16
        # the logits and their gradients are bf16: 2^-8 each of them
        assert abs(float(loss) - float((nll * scale).sum())) <= 2 ** -7 * float(nll.abs().sum()) and max(far[-1]) < 2 ** -6
    assert far[0][0] <= 1.02 * far[1][0] + 1e-4 and far[0][1] <= 1.02 * far[1][1] + 1e-4


@pytest.mark.parametrize("chunk", [96, 300])
def test_loss_lets_its_input_be_written_to(chunk):
    """Whatever waits for the backward is the loss's own: overwriting the hidden states before it changes no gradient."""
    from odc_b200 import ops
    torch.manual_seed(0)
    h0, w = torch.randn(300, 256, device="cuda").bfloat16(), torch.randn(1032, 256, device="cuda").bfloat16().requires_grad_()
    labels = torch.randint(0, 1032, (300,), device="cuda")
    grads = []
    for write in (False, True):
        leaf = h0.clone().requires_grad_()
        h = leaf * 1
        loss = ops.linear_cross_entropy(h, w, labels, chunk=chunk)
        if write:
            h.data.zero_()
            h.add_(1)
        grads.append(torch.autograd.grad(loss, [leaf, w]))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_weight_gradient_of_several_chunks_is_summed_in_one_order(monkeypatch):
    """Chunks are added to the fp32 matrix one after the other, each as one sum: the same bytes with and without a fixed order asked for."""
    from odc_b200 import ops
    torch.manual_seed(0)
    T, H, V = 6000, 256, 1024
    h = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    w = (0.05 * torch.randn(V, H, device="cuda")).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")
    grads = []
    for fixed in ("0", "1"):
        monkeypatch.setenv("ODC_DETERMINISTIC", fixed)
        grads.append(torch.autograd.grad(ops.linear_cross_entropy(h, w, labels, chunk=3000), [h, w]))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


@pytest.mark.parametrize("rows,cols", [(1, 8), (127, 72), (129, 264), (1001, 2560), (4096, 64)])
def test_bias_gradient_sums(ext, rows, cols):
    """Column sums, ragged in rows and in the 64 columns of a CTA: rounded once to bf16 from fp32 sums."""
    from odc_b200 import ops
    x, w = torch.randn(rows, 64, device="cuda").bfloat16(), torch.randn(cols, 64, device="cuda").bfloat16()
    b = torch.zeros(cols, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(rows, cols, device="cuda").bfloat16()
    db, = torch.autograd.grad(ops.linear(x, w, b), [b], dy)
    exact = dy.double().sum(0)
    # one rounding to bf16, and fp32 sums of `rows` terms of at most about 4
    assert ((db.double() - exact).abs() <= 2 ** -8 * exact.abs() + rows * 4 * 2 ** -22).all()


def test_bias_gradient_that_starts_off_a_16_byte_boundary():
    """Only the bias is trained, so no product looks at the gradient's start; column sums of 700 small whole numbers."""
    from odc_b200 import ops
    x, w = torch.randn(700, 512, device="cuda").bfloat16(), torch.randn(264, 512, device="cuda").bfloat16()
    b = torch.zeros(264, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    for skip in (0, 1, 4):
        dy = torch.randint(-1, 2, (700 * 264 + skip,), device="cuda").bfloat16()[skip:].view(700, 264)
        got, = torch.autograd.grad(ops.linear(x, w, b), [b], dy)
        assert torch.equal(got, dy.float().sum(0).bfloat16())


@pytest.mark.parametrize("dtype,N", [(torch.float32, 264), (torch.float16, 264), (torch.bfloat16, 12)])
def test_linear_on_library_products_in_other_types_and_widths(monkeypatch, dtype, N):
    """ODC_GEMM=cublas takes what the library takes; bias gradients of whole numbers are exact."""
    from odc_b200 import ops
    monkeypatch.setenv("ODC_GEMM", "cublas")
    x, w = torch.randn(100, 64, device="cuda", dtype=dtype), torch.randn(N, 64, device="cuda", dtype=dtype, requires_grad=True)
    b = torch.randn(N, device="cuda", dtype=dtype, requires_grad=True)
    dy = torch.randint(-1, 2, (100, N), device="cuda").to(dtype)
    y = ops.linear(x, w, b)
    assert y.dtype == dtype
    dw, db = torch.autograd.grad(y, [w, b], dy)
    assert torch.equal(db, dy.float().sum(0).to(dtype))
    assert torch.equal(dw, dy.t() @ x)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_lm_head_on_library_products_in_other_types(monkeypatch, dtype):
    """ODC_GEMM=cublas scores hidden states of any type; the logits are rounded to bf16 (2^-9 of values up to about 4)."""
    from odc_b200 import ops
    monkeypatch.setenv("ODC_GEMM", "cublas")
    h, w = torch.randn(100, 64, device="cuda", dtype=dtype), (torch.randn(512, 64, device="cuda") / 8).to(dtype)
    ids = torch.randint(0, 512, (100,), device="cuda")
    want = (h.double() @ w.double().t()).log_softmax(-1).gather(-1, ids[:, None])[:, 0]
    with torch.no_grad():
        torch.testing.assert_close(ops.linear_token_logprobs(h, w, ids).double(), want, rtol=0, atol=2e-2)
        torch.testing.assert_close(ops.linear_cross_entropy(h, w, ids).double(), -want.sum(), rtol=5e-3, atol=0)


def test_lm_head_refuses_a_chunk_or_temperature_of_zero():
    from odc_b200 import ops
    h, w = torch.randn(8, 64, device="cuda").bfloat16(), torch.randn(512, 64, device="cuda").bfloat16()
    ids = torch.randint(0, 512, (8,), device="cuda")
    for call in (ops.linear_cross_entropy, ops.linear_token_logprobs):
        with pytest.raises(ValueError):
            call(h, w, ids, chunk=0)
    with pytest.raises(ZeroDivisionError):
        ops.linear_token_logprobs(h, w, ids, temperature=0.0)


def test_linear_cross_entropy_matches_reference():
    from odc_b200 import ops
    from odc_b200.ops import reference as ref
    T, H, V = 700, 256, 1024
    h = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    w = (0.05 * torch.randn(V, H, device="cuda")).bfloat16().requires_grad_()
    labels = torch.randint(0, V, (T,), device="cuda")
    scale = torch.rand(T, device="cuda") / T
    loss = ops.linear_cross_entropy(h, w, labels, scale, chunk=256)
    (loss * 2.0).backward()
    hr, wr = h.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    lr_ = ref.linear_cross_entropy(hr, wr, labels, scale)
    (lr_ * 2.0).backward()
    torch.testing.assert_close(loss, lr_.detach(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(h.grad.float(), hr.grad, rtol=5e-2, atol=2e-4)
    torch.testing.assert_close(w.grad.float(), wr.grad, rtol=5e-2, atol=2e-4)


@pytest.mark.parametrize("temperature", [1.0, 0.7])
def test_linear_token_logprobs_one_chunk(temperature):
    """One chunk (weight gradient straight to bf16) against several (fp32 sums): apart by bf16 roundings of the gradient
    (2^-8 of its size), and the log-probabilities by nothing."""
    from odc_b200 import ops
    T, H, V = 384, 256, 1032
    h = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    w = (0.05 * torch.randn(V, H, device="cuda")).bfloat16().requires_grad_()
    ids, adv = torch.randint(0, V, (T,), device="cuda"), torch.randn(T, device="cuda")
    got = []
    for chunk in (128, T):
        lp = ops.linear_token_logprobs(h, w, ids, temperature, chunk=chunk)
        got.append((lp, *torch.autograd.grad(lp, [h, w], adv)))
    want = torch.log_softmax(h.double() @ w.double().t() / temperature, -1).gather(1, ids[:, None])[:, 0]
    torch.testing.assert_close(got[1][0].double(), want, rtol=0, atol=2e-2)  # bf16 logits of size 4: half a spacing is 2^-7
    for a, b in zip(*got):
        assert a.dtype == b.dtype
        assert ((a - b).float().norm() <= 2 ** -8 * b.float().norm()).item()


@pytest.mark.parametrize("temperature", [1.0, 0.7])
def test_linear_token_logprobs_matches_reference(temperature):
    """Per-token log-probabilities and both gradients against the fp32 statement of the same head; a 3-D input,
    a ragged last chunk and ignored positions included."""
    from odc_b200 import ops
    from odc_b200.ops import reference as ref
    B, S, H, V = 2, 333, 256, 1024
    h = torch.randn(B, S, H, device="cuda").bfloat16().requires_grad_()
    w = (0.05 * torch.randn(V, H, device="cuda")).bfloat16().requires_grad_()
    ids = torch.randint(0, V, (B, S), device="cuda")
    ids[0, :5] = -100
    adv = torch.randn(B, S, device="cuda")
    lp = ops.linear_token_logprobs(h, w, ids, temperature, chunk=256)
    assert lp.shape == ids.shape and lp.dtype == torch.float32
    (lp * adv).sum().backward()
    hr, wr = h.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    lpr = ref.linear_token_logprobs(hr.view(-1, H), wr, ids.view(-1), temperature).view(B, S)
    (lpr * adv).sum().backward()
    assert float(lp[0, :5].abs().max()) == 0.0
    torch.testing.assert_close(lp, lpr.detach(), rtol=2e-2, atol=3e-2)
    torch.testing.assert_close(h.grad.float(), hr.grad, rtol=5e-2, atol=3e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, rtol=5e-2, atol=5e-2)
    assert float(h.grad[0, :5].float().abs().max()) == 0.0


# ------------------------------------------------------------------------------------ fused compute + comm
@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("T,n_out,k_in", [(512, 256, 256), (1000, 768, 264), (4096, 2048, 2048)])
def test_wgrad_scatter_emulated_ranks(ext, world, T, n_out, k_in):
    """dW = dY^T X reduced straight into per-owner fp32 accumulators (owners emulated by local buffers)."""
    torch.manual_seed(T + n_out)
    rows_per = (n_out + world - 1) // world
    off = 64  # the parameter starts 64 elements into each accumulator
    accs = [torch.zeros(off + rows_per * k_in + 32, device="cuda") for _ in range(world)]
    ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
    want = torch.zeros(n_out, k_in, device="cuda")
    for producer in range(2):  # two emulated producers add into the same owners
        dy = torch.randn(T, n_out, device="cuda").bfloat16()
        x = torch.randn(T, k_in, device="cuda").bfloat16()
        ext.gemm_wgrad_scatter(dy, x, _table(accs), _table(ctrs), off, rows_per, 0.5)
        want += 0.5 * (dy.float().t() @ x.float())
    torch.cuda.synchronize()
    assert ext.kernel_status()[0].item() == 0
    for r in range(world):
        rows = max(0, min(rows_per, n_out - r * rows_per))
        got = accs[r][off:off + rows * k_in].view(rows, k_in)
        torch.testing.assert_close(got, want[r * rows_per:r * rows_per + rows], rtol=2e-2, atol=2e-2 * math.sqrt(T))
        assert float(accs[r][:off].abs().sum()) == 0.0 and float(accs[r][off + rows_per * k_in:].abs().sum()) == 0.0
        assert int(ctrs[r][0]) == 2


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("M,N,K", [(256, 512, 256), (1000, 1376, 512), (8192, 3072, 2048), (300, 264, 128)])
def test_gemm_gather_emulated_ranks(ext, world, M, N, K):
    """Y = X W^T with W assembled from row shards while the GEMM runs (owners emulated by local buffers)."""
    torch.manual_seed(M + N + K)
    rows_per = (N + world - 1) // world
    W = torch.randn(world * rows_per, K, device="cuda").bfloat16()
    shards = [W[r * rows_per:(r + 1) * rows_per].clone() for r in range(world)]
    x = torch.randn(M, K, device="cuda").bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    w_local = torch.zeros(N, K, dtype=torch.bfloat16, device="cuda")
    y = ext.gemm_gather(x, _table(shards), w_local, bias, rows_per, (world - 1) if world > 2 else 1 % world)
    torch.cuda.synchronize()
    assert ext.kernel_status()[0].item() == 0, ext.kernel_status().tolist()
    assert torch.equal(w_local, W[:N])
    torch.testing.assert_close(y.float(), x.float() @ W[:N].float().t() + bias.float(), rtol=2e-2, atol=2e-2 * math.sqrt(K))


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("M,N,K", [(256, 512, 256), (1000, 1376, 512), (8192, 3072, 2048), (300, 264, 128)])
def test_gemm_gather_dgrad_emulated_ranks(ext, world, M, N, K):
    """dX = dY W with W's rows (the reduction dimension) assembled from shards while the GEMM runs."""
    torch.manual_seed(M + N + K + 1)
    rows_per = (N + world - 1) // world
    W = (0.1 * torch.randn(world * rows_per, K, device="cuda")).bfloat16()
    shards = [W[r * rows_per:(r + 1) * rows_per].clone() for r in range(world)]
    dy = torch.randn(M, N, device="cuda").bfloat16()
    w_local = torch.zeros(N, K, dtype=torch.bfloat16, device="cuda")
    dx = ext.gemm_gather_dgrad(dy, _table(shards), w_local, rows_per, (world * 5 + 3) % world if world > 2 else world - 1)
    torch.cuda.synchronize()
    assert ext.kernel_status()[0].item() == 0, ext.kernel_status().tolist()
    assert torch.equal(w_local, W[:N])
    torch.testing.assert_close(dx.float(), dy.float() @ W[:N].float(), rtol=2e-2, atol=2e-2 * math.sqrt(N) * 0.1)


def test_linear_with_fused_residual():
    from odc_b200 import ops
    x = torch.randn(300, 512, device="cuda").bfloat16().requires_grad_()
    w = (0.05 * torch.randn(768, 512, device="cuda")).bfloat16().requires_grad_()
    res = torch.randn(300, 768, device="cuda").bfloat16().requires_grad_()
    y = ops.linear(x, w, None, residual=res)
    dy = torch.randn_like(y)
    y.backward(dy)
    want = x.detach().float() @ w.detach().float().t() + res.detach().float()
    torch.testing.assert_close(y.float(), want, rtol=2e-2, atol=5e-2)
    assert torch.equal(res.grad, dy)


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("T,n_out,k_in", [(512, 1024, 256), (1000, 2048, 264), (4096, 2048, 2048)])
def test_wgrad_scatter_tma_emulated_ranks(ext, world, T, n_out, k_in):
    """Same contract as the red.add variant, output through smem staging + TMA reduce-add (owners emulated locally)."""
    torch.manual_seed(T + n_out)
    rows_per = (n_out + world - 1) // world
    rows_per = (rows_per + 127) // 128 * 128
    off = 64
    accs = [torch.zeros(off + rows_per * k_in + 32, device="cuda") for _ in range(world)]
    ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
    want = torch.zeros(world * rows_per, k_in, device="cuda")
    for producer in range(2):
        dy = torch.randn(T, n_out, device="cuda").bfloat16()
        x = torch.randn(T, k_in, device="cuda").bfloat16()
        # the producer's position in the group only rotates the order in which the owners' tiles are produced
        assert ext.gemm_wgrad_scatter_tma(dy, x, [a.data_ptr() for a in accs], _table(ctrs), off, rows_per, 0.5,
                                          (producer * 5 + 1) % world)
        want[:n_out] += 0.5 * (dy.float().t() @ x.float())
    torch.cuda.synchronize()
    assert ext.kernel_status()[0].item() == 0
    for r in range(world):
        got = accs[r][off:off + rows_per * k_in].view(rows_per, k_in)
        torch.testing.assert_close(got, want[r * rows_per:(r + 1) * rows_per], rtol=2e-2, atol=2e-2 * math.sqrt(T))
        assert float(accs[r][:off].abs().sum()) == 0.0 and float(accs[r][off + rows_per * k_in:].abs().sum()) == 0.0
        assert int(ctrs[r][0]) == 2
    # ineligible split (rows per owner not a multiple of 128): the entry point declines, nothing is launched
    assert not ext.gemm_wgrad_scatter_tma(dy, x, [a.data_ptr() for a in accs], _table(ctrs), off, 100, 1.0)


def test_scatter_accumulate_bulk_path_matches(ext):
    """The opt-in bulk (TMA) scatter path gives the same sums; run in a child process so the switch is seen at first use."""
    import subprocess, sys, os, textwrap
    code = textwrap.dedent("""
        import torch, sys
        sys.path.insert(0, %r)
        from odc_b200 import _ext
        ext = _ext.load()
        world, n = 4, 1 << 18
        accs = [torch.zeros(n, device="cuda") for _ in range(world)]
        ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
        tab = lambda ts: torch.tensor([t.data_ptr() for t in ts], dtype=torch.int64, device="cuda")
        xs = [torch.randint(-4, 5, (world, n), device="cuda").float() for _ in range(world)]
        st = torch.zeros(4, dtype=torch.int32, device="cuda")
        for me in range(world):
            ext.scatter_accumulate(xs[me], tab(accs), tab(ctrs), n, torch.float32, me, 1.0, False, st)
        torch.cuda.synchronize()
        want = torch.stack(xs).sum(0)
        assert all(torch.equal(accs[p], want[p]) for p in range(world))
        assert all(int(c[0]) == world for c in ctrs) and int(st[0]) == 0
        print("BULK_OK")
    """ % os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, ODC_SCATTER_BULK="1"), capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and "BULK_OK" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_scatter_accumulate_segments_emulated_ranks(ext, world, dtype):
    """Reduction straight from a list of gradient tensors: same result as flattening them rank-major first."""
    torch.manual_seed(world)
    shapes = [(1024, 512), (512,), (300, 96), (7, 5), (world * 3 + 1, 64), (2048, 2048)]
    grads = [torch.randn(*s, device="cuda").to(dtype) for s in shapes]
    chunks, offsets, o = [], [], 0
    for g in grads:
        rows = -(-g.shape[0] // world)
        c = rows * (g.numel() // g.shape[0])
        chunks.append(c)
        offsets.append(o)
        o += c
    accs = [torch.zeros(o + 16, device="cuda") for _ in range(world)]
    ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
    for _ in range(2):
        assert ext.scatter_accumulate_segments(grads, chunks, offsets, _table(accs), _table(ctrs), torch.float32, 1 % world, 0.5)
    torch.cuda.synchronize()
    for r in range(world):
        want = torch.zeros(o + 16, device="cuda")
        for g, c, off in zip(grads, chunks, offsets):
            piece = g.reshape(-1)[r * c:(r + 1) * c].float()
            want[off:off + piece.numel()] += 2 * 0.5 * piece
        torch.testing.assert_close(accs[r], want, rtol=1e-6, atol=1e-6)
        assert int(ctrs[r][0]) == 2
    # lists this path does not take are refused without a launch
    assert not ext.scatter_accumulate_segments([grads[0]] * 33, [chunks[0]] * 33, [0] * 33, _table(accs), _table(ctrs),
                                               torch.float32, 0, 1.0)
    assert not ext.scatter_accumulate_segments(grads, chunks, offsets, _table(accs), _table(ctrs), torch.bfloat16, 0, 1.0)


# ------------------------------------------------------------------------------------ debug bounds checks
def test_debug_bounds_refuse_a_short_declared_region(ext):
    """ODC_DEBUG_BOUNDS launches: a row longer than the DECLARED region is refused on valid memory.

    Every buffer here is fully allocated, only the declared length is made too short, so nothing out of range
    is ever touched; a refused launch leaves the destination untouched and reports through the status word.
    """
    world, n = 2, 4096
    from odc_b200.runtime.status import ERR_BOUNDS, ERR_PEER_INDEX
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    # gather
    shards = [torch.ones(n, device="cuda").bfloat16() * (r + 1) for r in range(world)]
    out = torch.zeros(world, n, dtype=torch.bfloat16, device="cuda")
    ext.gather(out, _table(shards), n, torch.bfloat16, 0, True, status, n - 8)
    torch.cuda.synchronize()
    assert int(status[0]) == ERR_BOUNDS and float(out.abs().sum()) == 0
    status.zero_()
    ext.gather(out, _table(shards), n, torch.bfloat16, 5, True, status, n)      # start index outside the group
    torch.cuda.synchronize()
    assert int(status[0]) == ERR_PEER_INDEX and float(out.abs().sum()) == 0
    status.zero_()
    ext.gather(out, _table(shards), n, torch.bfloat16, 1, True, status, n)      # exact fit passes
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and torch.equal(out, torch.stack(shards))
    # scatter_accumulate (fp32 and bf16 sources, fp32 and bf16 accumulators)
    for in_dtype, acc_dtype in [(torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                (torch.bfloat16, torch.bfloat16)]:
        accs = [torch.zeros(n, dtype=acc_dtype, device="cuda") for _ in range(world)]
        ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
        x = torch.ones(world, n, device="cuda").to(in_dtype)
        status.zero_()
        ext.scatter_accumulate(x, _table(accs), _table(ctrs), n, acc_dtype, 0, 1.0, True, status, n - 4)
        torch.cuda.synchronize()
        assert int(status[0]) == ERR_BOUNDS
        assert all(float(a.float().abs().sum()) == 0 for a in accs)
        assert all(int(c[0]) == 1 for c in ctrs)   # the owners are not left waiting for the refused contribution
        status.zero_()
        ext.scatter_accumulate(x, _table(accs), _table(ctrs), n, acc_dtype, 0, 1.0, True, status, n)
        torch.cuda.synchronize()
        assert int(status[0]) == 0 and all(float(a.float().sum()) == n for a in accs)
    # segmented scatter: the second tensor would end past the declared accumulator length
    accs = [torch.zeros(3 * n, device="cuda") for _ in range(world)]
    ctrs = [torch.zeros(8, dtype=torch.int64, device="cuda") for _ in range(world)]
    grads = [torch.ones(world * n, device="cuda"), torch.ones(world * 2 * n, device="cuda")]
    status.zero_()
    assert ext.scatter_accumulate_segments(grads, [n, 2 * n], [0, n], _table(accs), _table(ctrs), torch.float32, 0, 1.0,
                                           True, status, 3 * n - 4)
    torch.cuda.synchronize()
    assert int(status[0]) == ERR_BOUNDS and all(float(a.sum()) == 0 for a in accs)
    status.zero_()
    assert ext.scatter_accumulate_segments(grads, [n, 2 * n], [0, n], _table(accs), _table(ctrs), torch.float32, 0, 1.0,
                                           True, status, 3 * n)
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and all(float(a.sum()) == 3 * n for a in accs)


def test_posted_counts_and_bounded_wait(ext):
    """One-sided dispatch-count exchange, with the producers emulated by separate posts into one owner's slots."""
    nprod = 5
    slots = torch.zeros(8, dtype=torch.int64, device="cuda")
    ctr = torch.zeros(8, dtype=torch.int64, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    expected = torch.zeros(1, dtype=torch.int64, device="cuda")
    counts = [3, 0, 7, 1, 2]
    for p, c in enumerate(counts):
        ext.post_counts([slots.data_ptr() + 8 * p], [c], 1, 0)
    ctr[0] = sum(counts)
    ext.wait_posted(slots, nprod, 1, ctr, 500, status, expected)
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and int(expected[0]) == sum(counts)
    assert [int(v) >> 32 for v in slots[:nprod]] == [1] * nprod
    # a synchronisation that one producer never posts for: the wait runs out and names the producer
    for p, c in enumerate(counts[:-1]):
        ext.post_counts([slots.data_ptr() + 8 * p], [c + 1], 2, 0)
    ext.wait_posted(slots, nprod, 2, ctr, 50, status, expected)
    torch.cuda.synchronize()
    assert status[:3].tolist() == [1, 1000 + nprod - 1, 1]
    # all postings there, but fewer arrivals than announced: the arrival wait runs out instead
    status.zero_()
    ext.post_counts([slots.data_ptr() + 8 * (nprod - 1)], [counts[-1] + 1], 2, 0)
    ext.wait_posted(slots, nprod, 2, ctr, 50, status, expected)
    torch.cuda.synchronize()
    assert status[:3].tolist() == [1, 0, sum(counts)] and int(expected[0]) == sum(counts) + nprod


def test_rmsnorm_residual_backward_fuses_the_residual_gradient():
    """(norm(x), x): the gradient of the pass-through output is added inside the norm's backward kernel."""
    from odc_b200 import ops
    rows, cols = 777, 2048
    x = torch.randn(rows, cols, device="cuda").bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(cols, device="cuda")).bfloat16().requires_grad_()
    y, xr = ops.rms_norm_residual(x, w, 1e-5)
    dy, dres = torch.randn_like(y), torch.randn_like(xr)
    torch.autograd.backward([y, xr], [dy, dres])
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    torch.autograd.backward([yf, xf * 1.0], [dy.float(), dres.float()])
    torch.testing.assert_close(y.float(), yf, rtol=2e-2, atol=2e-2)
    assert xr.data_ptr() == x.data_ptr()
    torch.testing.assert_close(x.grad.float(), xf.grad, rtol=2e-2, atol=3e-2)
    torch.testing.assert_close(w.grad.float(), wf.grad, rtol=2e-2, atol=rows ** 0.5 * 2e-2)
    # only the normalised branch is used: the pass-through gradient is absent
    x2 = x.detach().clone().requires_grad_()
    y2, _ = ops.rms_norm_residual(x2, w.detach(), 1e-5)
    y2.backward(dy)
    xg = x.detach().float().requires_grad_()
    (xg * torch.rsqrt(xg.pow(2).mean(-1, keepdim=True) + 1e-5) * w.detach().float()).backward(dy.float())
    torch.testing.assert_close(x2.grad.float(), xg.grad, rtol=2e-2, atol=3e-2)


@pytest.mark.parametrize("T,V,H,chunk", [(256, 264, 64, 4096), (700, 1000, 512, 300), (520, 8200, 256, 512), (900, 264, 64, 4096),
                                         (1700, 1000, 512, 800), (1000, 8200, 256, 777)])
@pytest.mark.parametrize("temperature", [1.0, 0.7])
def test_head_statistics_from_the_product(ext, T, V, H, chunk, temperature):
    """Softmax statistics of ragged tiles, in chunks (short ones take the passes over logits): log-probabilities, loss and
    both gradients; ignored and weightless rows; a NaN row stays one row."""
    from odc_b200 import ops
    torch.manual_seed(T + V)
    h = (2 * torch.randn(T, H, device="cuda")).bfloat16().requires_grad_()
    w = (torch.randn(V, H, device="cuda") * H ** -0.5).bfloat16().requires_grad_()
    ids = torch.randint(0, V, (T,), device="cuda")
    ids[3], ids[5], ids[7] = -100, V - 1, 0
    dlogp = torch.randn(T, device="cuda")
    lp = ops.linear_token_logprobs(h, w, ids, temperature, chunk=chunk)
    dh, dw = torch.autograd.grad(lp, [h, w], dlogp)
    h64, w64 = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    keep = ids >= 0
    want = torch.where(keep, ((h64 @ w64.t()) / temperature).log_softmax(-1).gather(1, ids.clamp_min(0)[:, None])[:, 0], 0.0)
    wh, ww = torch.autograd.grad(want, [h64, w64], dlogp.double())
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    # logits are rounded to bf16 (at most 2^-8 of each), the label's and those of the row's sum: 2e-2 of a gradient's weight
    size = (h64 @ w64.t()).detach().abs()
    bound = 2 ** -8 * (size.gather(1, ids.clamp_min(0)[:, None])[:, 0] + size.amax(1)) / temperature + 1e-4
    assert ((lp.double() - want).abs() <= bound).all() and lp[3].item() == 0.0
    assert rel(dh, wh) < 1.5e-2 and rel(dw, ww) < 1.5e-2
    weight = torch.rand(T, device="cuda")
    weight[9] = 0.0
    loss = ops.linear_cross_entropy(h, w, ids, weight, chunk=chunk)
    gh, gw = torch.autograd.grad(loss, [h, w])
    logp = (h64 @ w64.t()).log_softmax(-1).gather(1, ids.clamp_min(0)[:, None])[:, 0]
    want = -(torch.where(keep, logp, 0.0) * weight.double()).sum()
    wh, ww = torch.autograd.grad(want, [h64, w64])
    assert abs(loss.item() - want.item()) < 1e-3 * abs(want.item())
    assert rel(gh, wh) < 1.5e-2 and rel(gw, ww) < 1.5e-2
    assert gh[3].abs().max().item() == 0.0 and gh[9].abs().max().item() == 0.0
    bad = h.detach().clone()
    bad[11] = float("nan")
    with torch.no_grad():
        out = ops.linear_token_logprobs(bad, w, ids, temperature, chunk=chunk)
    assert out[11].isnan() and out[12:].isfinite().all() and out[:11].isfinite().all()
    bad.requires_grad_()
    loss = ops.linear_cross_entropy(bad, w, ids, weight, chunk=chunk)
    gh, = torch.autograd.grad(loss, bad)
    assert loss.isnan() and gh[11].isnan().all() and gh[12:].isfinite().all() and gh[:11].isfinite().all()
    assert ext.kernel_status()[0].item() == 0


def test_passes_over_logits_of_minus_infinity(ext):
    """Eight logits of -inf in one thread's hands, at the start of its row or all of it, weigh nothing."""
    torch.manual_seed(3)
    T, V = 5, 16648
    x = torch.randn(T, V, device="cuda").bfloat16()
    x[0, 256:512], x[1, :8], x[2, 8:], x[3, 8192:8208] = (float("-inf"),) * 4
    ids = torch.tensor([3, 9, 5, 8300, 7], device="cuda")
    want = x.double().log_softmax(-1)
    out, loss, grad = torch.empty(T, device="cuda"), torch.zeros((), device="cuda"), x.clone()
    ext.token_logprobs(x, ids, out, -100, 1.0)
    ext.ce_fwd_bwd(grad, ids, None, loss, -100, 1.0)
    picked = want[torch.arange(T), ids]
    # fp32 sums of V exponentials, each to a few 2^-22: far below 1e-4; gradients are rounded to bf16 (2^-8 of their size)
    assert (out.double() - picked).abs().max().item() < 1e-4 and abs(loss.item() + picked.sum().item()) < 1e-3
    d = want.exp() - torch.nn.functional.one_hot(ids, V)
    assert ((grad.double() - d).abs() <= 2 ** -8 * d.abs() + 1e-6).all()


@pytest.mark.parametrize("T,V", [(256, 1000), (800, 1000), (1000, 2056)])
def test_head_statistics_of_infinite_logits(ext, T, V):
    """Logits of -inf beside finite ones, over a whole tile of 256 words and in single places: they have no weight, and nothing
    else changes.  A row of nothing but -inf has no probabilities, as a softmax in 64 bits has none."""
    from odc_b200 import ops
    torch.manual_seed(T + V)
    h = torch.randn(T, 64, device="cuda").bfloat16()
    w = (torch.randn(V, 64, device="cuda") / 8).bfloat16()
    gone = torch.zeros(V, dtype=torch.bool, device="cuda")
    gone[256:512] = True
    gone[torch.arange(3, V, 97, device="cuda")] = True
    h[:, :2], w[:, :2] = 0.0, 0.0
    h[5, 0], h[40, 0], h[7, 1] = 1e20, 1e20, 1e20     # their logits: -1e40 where a word has -1e20 in the same place
    w[gone, 0], w[:, 1] = -1e20, -1e20
    h.requires_grad_(), w.requires_grad_()
    ids = (~gone).nonzero()[:, 0][torch.randint(0, int((~gone).sum()), (T,), device="cuda")]
    lp = ops.linear_token_logprobs(h, w, ids)
    logits = h.detach().double() @ w.detach().double().t()
    logits = torch.where(logits < -1e38, float("-inf"), logits)
    want = logits.log_softmax(-1)
    keep = torch.arange(T, device="cuda") != 7
    # logits up to about 6 are rounded to bf16 (2^-8 of their size)
    assert (lp.double() - want[torch.arange(T), ids])[keep].abs().max().item() < 2 ** -8 * 12 and lp[7].isnan()
    weight = torch.ones(T, device="cuda")
    weight[7] = 0.0                                    # ignored in the loss: no NaN gets into it or the gradients
    loss = ops.linear_cross_entropy(h, w, ids, weight)
    gh, gw = torch.autograd.grad(loss, [h, w])
    d = (want.exp() - torch.nn.functional.one_hot(ids, V).double()) * keep[:, None]
    d = torch.where(keep[:, None], d, 0.0)
    assert abs(loss.item() + want[torch.arange(T), ids][keep].sum().item()) < 1e-3 * loss.item()
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    assert rel(gh[:, 2:], (d @ w.detach().double())[:, 2:]) < 1.5e-2
    assert rel(gw[:, 2:], (d.t() @ h.detach().double())[:, 2:]) < 1.5e-2
    assert ext.kernel_status()[0].item() == 0


@pytest.mark.parametrize("T,H,F", [(256, 64, 256), (300, 512, 264), (1000, 264, 1544), (16000, 256, 512), (24, 256, 512)])
def test_mlp_matches_its_parts(ext, T, H, F):
    """One function against linear(swiglu(linear)): ragged tiles of either dimension, more tiles than pairs, and a shape
    that the fused epilogue does not take."""
    from odc_b200 import ops
    torch.manual_seed(T + H + F)
    x = torch.randn(T, H, device="cuda").bfloat16().requires_grad_()
    gu = (torch.randn(2 * F, H, device="cuda") * H ** -0.5).bfloat16().requires_grad_()
    down = (torch.randn(H, F, device="cuda") * F ** -0.5).bfloat16().requires_grad_()
    res, dy = torch.randn(T, H, device="cuda").bfloat16().requires_grad_(), torch.randn(T, H, device="cuda").bfloat16()
    y = ops.mlp(x, gu, down, res)
    got = torch.autograd.grad(y, [x, gu, down, res], dy)
    parts = ops.linear(ops.linear_swiglu(x, gu), down, residual=res)
    want = torch.autograd.grad(parts, [x, gu, down, res], dy)
    assert ext.kernel_status()[0].item() == 0
    assert torch.equal(y, parts) and torch.equal(got[3], dy)
    for g, w in zip(got[:3], want[:3]):   # the same roundings; only the fp32 sums of a divided product may be in another order
        assert ((g.float() - w.float()).norm() / w.float().norm()).item() < 1e-3
    # the projection's gradient by itself, edges of both halves included
    gate_up = ops.linear(x, gu).detach()
    one, two = ext.swiglu_product_bwd(dy, down.detach(), gate_up), ext.swiglu_bwd(dy @ down.detach(), gate_up)
    assert ((one.float() - two.float()).norm() / two.float().norm()).item() < 1e-2


def test_log_probabilities_alone_hold_no_logits():
    """Forward only, the product leaves row statistics (8 bytes per 256 words) and the logits are never written: no scratch for
    them is held, except for a last chunk below a tile of rows, which takes the passes over logits."""
    from odc_b200 import ops
    T, V, H, chunk = 2124, 8192, 256, 1024         # chunks of 1024, 1024 and 76 rows
    h, w = torch.randn(T, H, device="cuda").bfloat16(), torch.randn(V, H, device="cuda").bfloat16()
    ids = torch.randint(0, V, (T,), device="cuda")
    run = lambda n: ops.linear_token_logprobs(h[:n], w, ids[:n], chunk=chunk)
    with torch.no_grad():
        for n, limit in ((2048, 1 << 20), (T, (1 << 20) + 76 * V * 2)):
            run(n)
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            held = torch.cuda.memory_allocated()
            out = run(n)
            torch.cuda.synchronize()
            assert torch.cuda.max_memory_allocated() - held < limit
            want = (h[:n].double() @ w.double().t()).log_softmax(-1).gather(1, ids[:n, None])[:, 0]
            # logits around 100 are rounded to bf16: 2^-8 of their size
            assert (out.double() - want).abs().max().item() < 2 ** -8 * 200
        for chunk, error in ((0, ValueError), (-1, RuntimeError)):
            for n in (0, T):
                with pytest.raises(error):
                    run(n)
