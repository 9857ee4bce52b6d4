"""Kernel-level GPU checks through the C-ABI microbenchmark entry points: the tcgen05 GEMM in
all operand layouts against an FP32 product, attention and cross-entropy against plain PyTorch."""
import ctypes

import numpy as np
import pytest
import torch

from turbogpt_b200 import load_library
from helpers import max_relative

pytestmark = pytest.mark.gpu
BACKWARD_ON_TENSOR_CORES = True


def gemm(lib, a, a_strides, b, b_strides, m, n, k, out_fp32, tensor_cores):
    c = torch.zeros(m, n, device="cuda", dtype=torch.float32 if out_fp32 else torch.bfloat16)
    status = lib.tg_ex_gemm(a.data_ptr(), *a_strides, b.data_ptr(), *b_strides, c.data_ptr(), n, m, n, k,
                            int(out_fp32), int(tensor_cores), None)
    assert status == 0, lib.tg_error().decode()
    torch.cuda.synchronize()
    return c.float().cpu().numpy()


def operands(m, n, k, a_mn, b_mn, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    a = torch.randn(m, k, generator=g).bfloat16()
    b = torch.randn(n, k, generator=g).bfloat16()
    expected = (a.float() @ b.float().T).numpy()
    a_dev = (a.T.contiguous() if a_mn else a).cuda()   # MN-major: stored [k, m]
    b_dev = (b.T.contiguous() if b_mn else b).cuda()
    a_strides = (1, m) if a_mn else (k, 1)
    b_strides = (1, n) if b_mn else (k, 1)
    return a_dev, a_strides, b_dev, b_strides, expected


# forward (K-major, K-major), input gradient (K-major, MN-major), weight gradient (MN, MN)
LAYOUTS = [(False, False), (False, True), (True, True), (True, False)]


@pytest.mark.parametrize("a_mn,b_mn", LAYOUTS)
@pytest.mark.parametrize("m,n,k", [(128, 64, 64), (256, 256, 128), (384, 192, 320), (1000, 264, 200),
                                   (128, 768, 4096), (4096, 2304, 768),
                                   (200, 136, 8192)])  # ragged edges with many K splits (added by their own kernel)
def test_tensor_core_gemm_matches_fp32_product(a_mn, b_mn, m, n, k):
    lib = load_library()
    if a_mn and m % 8:
        pytest.skip("an MN-major A needs a multiple of 8 rows")
    a, sa, b, sb, expected = operands(m, n, k, a_mn, b_mn)
    for out_fp32 in (True, False):
        got = gemm(lib, a, sa, b, sb, m, n, k, out_fp32, True)
        # FP32 accumulation of exact BF16 products: only summation order differs.
        tolerance = 1e-5 if out_fp32 else 4e-3
        assert max_relative(got, expected) <= tolerance, (m, n, k, a_mn, b_mn, out_fp32)
        simt = gemm(lib, a, sa, b, sb, m, n, k, out_fp32, False)
        assert max_relative(simt, expected) <= tolerance


# (tile columns, K splits, CTA pair) with K-major and with MN-major B, and how many rounds of tiles a block takes on 148 SMs.
TILE_FORMS = [
    ((129, 72, 72), (64, 1, 0), (64, 1, 0), 1), ((4100, 264, 72), (128, 1, 0), (128, 1, 0), 1),
    ((4100, 520, 72), (192, 1, 0), (192, 1, 0), 1), ((4100, 776, 72), (256, 1, 0), (256, 1, 0), 1),
    ((20000, 72, 72), (64, 1, 0), (64, 1, 0), 3), ((20000, 72, 200), (128, 1, 0), (128, 1, 0), 2),
    ((9000, 520, 72), (192, 1, 0), (192, 1, 0), 2), ((33000, 200, 72), (256, 1, 0), (256, 1, 0), 2),
    ((4100, 264, 1032), (128, 1, 1), (128, 1, 1), 1), ((2050, 1544, 520), (256, 1, 1), (256, 1, 1), 1),
    ((4100, 520, 3080), (192, 1, 1), (256, 1, 1), 1), ((4100, 776, 3080), (256, 1, 1), (256, 1, 1), 1),
    ((16400, 136, 3080), (192, 1, 1), (192, 1, 0), 1),
    ((20000, 72, 1032), (128, 1, 1), (128, 1, 1), 2), ((33000, 200, 520), (256, 1, 1), (256, 1, 1), 2),
    ((129, 72, 3080), (64, 6, 0), (64, 6, 0), 1), ((129, 2056, 3080), (128, 4, 0), (128, 4, 0), 1),
    ((2305, 272, 8008), (192, 3, 1), (128, 2, 1), 1)]  # the last of two or three blocks adds their parts itself


def test_tile_forms_are_what_the_schedule_chooses():
    for (m, n, k), *forms, rounds in TILE_FORMS:
        for b_mn, form in enumerate(forms):
            plan = (ctypes.c_int32 * 4)()
            assert load_library().tg_ex_gemm_schedule(k, 1, *((1, n) if b_mn else (k, 1)), n, m, n, k, 1, 0, 0, 148, plan) == 0
            assert tuple(plan)[:3] == form, (m, n, k, b_mn)
            columns, splits, pair = form
            tiles = -(-m // (256 if pair else 128)) * -(-n // columns) * splits
            assert -(-tiles // (74 if pair else 148)) == rounds


@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("m,n,k", [form[0] for form in TILE_FORMS])
def test_products_of_every_tile_form_at_their_edges(m, n, k, b_mn):
    """The choices of the schedule, with partial tiles in every dimension, against 64 bits: FP32 sums of k exact products, then one
    BF16 rounding; and with a second tensor (never with K cut), two FP32 roundings of either term before it."""
    lib = load_library()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a, b = (torch.randn(rows, k, generator=g, device="cuda").bfloat16() for rows in (m, n))
    stored = b.T.contiguous() if b_mn else b
    c, scaled = (torch.empty(m, n, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    r = torch.randn(m, n, generator=g, device="cuda").bfloat16()
    strides = (1, n) if b_mn else (k, 1)
    assert lib.tg_ex_gemm(a.data_ptr(), k, 1, stored.data_ptr(), *strides, c.data_ptr(), n, m, n, k, 0, 1, None) == 0, lib.tg_error()
    assert lib.tg_ex_gemm_batched(a.data_ptr(), k, 1, 0, stored.data_ptr(), *strides, 0, scaled.data_ptr(), n, 0, r.data_ptr(), .5, 3.,
                                  m, n, k, 1, 0, None) == 0, lib.tg_error()
    torch.cuda.synchronize()
    expected, magnitude = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    bound = k * 2.0 ** -24 * magnitude
    assert ((c.double() - expected).abs() <= bound + 2.0 ** -8 * expected.abs()).all()
    second = .5 * expected + 3. * r.double()
    assert ((scaled.double() - second).abs() <=
            .5 * bound + 2.0 ** -22 * (.5 * expected.abs() + 3. * r.double().abs()) + 2.0 ** -8 * second.abs()).all()
    assert lib.tg_ex_last_device_error(None) == 0


def test_batches_of_more_matrices_than_a_launch_takes():
    """2^20 tiles to a launch: matrices on both sides of the border, the second tensor's too, against 64 bits.  Neighbouring matrices share
    all but 16 bytes."""
    lib, batch, n, k = load_library(), 2 ** 20 + 5, 64, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b = (torch.randn(8 * batch + size, generator=g, device="cuda").bfloat16() for size in (k, n * k))
    r = torch.randn(batch, n, generator=g, device="cuda").bfloat16()
    c, scaled = (torch.full((batch, n), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    for out, second in ((c, None), (scaled, r.data_ptr())):
        assert lib.tg_ex_gemm_batched(a.data_ptr(), k, 1, 8, b.data_ptr(), k, 1, 8, out.data_ptr(), n, n, second, .5, 3.,
                                      1, n, k, batch, 0, None) == 0, lib.tg_error()
    torch.cuda.synchronize()
    assert torch.isfinite(c).all() and torch.isfinite(scaled).all()
    for first in (0, 2 ** 20 - 500):
        some = slice(first, first + 505)
        x, w = a.as_strided((505, 1, k), (8, k, 1), 8 * first).double(), b.as_strided((505, n, k), (8, k, 1), 8 * first).double()
        exact, bound = ((x @ w.mT)[:, 0], k * 2.0 ** -24 * (x.abs() @ w.abs().mT)[:, 0])
        assert ((c[some].double() - exact).abs() <= bound + 2.0 ** -8 * exact.abs()).all()
        expected = .5 * exact + 3. * r[some].double()
        assert ((scaled[some].double() - expected).abs() <=
                .5 * bound + 2.0 ** -22 * (.5 * exact.abs() + 3. * r[some].double().abs()) + 2.0 ** -8 * expected.abs()).all()
    assert lib.tg_ex_last_device_error(None) == 0


@pytest.mark.parametrize("m,n,k,b_mn", [
    *((m, n, k, b_mn) for k in (64, 72, 192, 320, 1544)  # shorter than the ring of half an SM, as long, round after round
      for m, n, b_mn in ((320, 320, False), (320, 320, True), (129, 72, True), (64, 64, False),  # 64 columns, four stages
                         (320, 1928, False), (320, 1928, True))),                                # 128 columns, three stages
    (129, 72, 3080, True), (320, 320, 3080, False)])                                             # K cut in six, in four
def test_batched_products_in_half_an_sm(m, n, k, b_mn):
    """Partial tiles in every dimension against 64 bits, both epilogues; two such products run at once, so that blocks of both
    share SMs; and with an SM for each tile, bit for bit."""
    lib, batch = load_library(), 3
    plan = (ctypes.c_int32 * 4)()
    assert lib.tg_ex_gemm_schedule(k, 1, *((1, n) if b_mn else (k, 1)), n, m, n, k, batch, 0, 1, 148, plan) == 0 and plan[3] == 1
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a, b, r = (torch.randn(batch, *shape, generator=g, device="cuda").bfloat16() for shape in ((m, k), (n, k), (m, n)))
    stored = b.transpose(1, 2).contiguous() if b_mn else b
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()

    def product(out, second, beside, stream):
        assert lib.tg_ex_gemm_batched(a.data_ptr(), k, 1, m * k, stored.data_ptr(), *((1, n) if b_mn else (k, 1)), n * k,
                                      out.data_ptr(), n, m * n, second, 2.0315, -4.775, m, n, k, batch, beside,
                                      stream.cuda_stream) == 0, lib.tg_error()

    plain, scaled = ([torch.full((batch, m, n), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(9)] for _ in range(2))
    torch.cuda.synchronize()
    for p, s in zip(plain[:8], scaled[:8]):
        product(p, None, 1, streams[0])
        product(s, r.data_ptr(), 1, streams[1])
    product(plain[8], None, 0, streams[0])
    product(scaled[8], r.data_ptr(), 0, streams[1])
    torch.cuda.synchronize()
    exact, magnitude = a.double() @ b.double().transpose(1, 2), a.double().abs() @ b.double().abs().transpose(1, 2)
    # FP32 sums of k exact products, then for the second form two FP32 roundings of either term, and one to BF16
    bound = k * 2.0 ** -24 * magnitude
    assert ((plain[0].double() - exact).abs() <= bound + 2.0 ** -8 * exact.abs()).all()
    expected = 2.0315 * exact - 4.775 * r.double()
    assert ((scaled[0].double() - expected).abs() <=
            2.0315 * bound + 2.0 ** -22 * (2.0315 * exact.abs() + 4.775 * r.double().abs()) + 2.0 ** -8 * expected.abs()).all()
    for p, s in zip(plain[1:], scaled[1:]):
        assert torch.equal(p, plain[0]) and torch.equal(s, scaled[0])
    assert lib.tg_ex_last_device_error(None) == 0


def test_split_k_weight_gradient_is_deterministic():
    lib = load_library()
    a, sa, b, sb, expected = operands(768, 768, 16384, True, True, seed=3)
    first = gemm(lib, a, sa, b, sb, 768, 768, 16384, True, True)
    assert max_relative(first, expected) <= 2e-5
    for _ in range(3):
        np.testing.assert_array_equal(first, gemm(lib, a, sa, b, sb, 768, 768, 16384, True, True))


def test_cross_entropy_matches_torch():
    lib = load_library()
    rows = 4096 + 3
    g = torch.Generator().manual_seed(0)
    logits = torch.randn(rows, 256, generator=g).bfloat16()
    targets = torch.randint(0, 256, (rows,), generator=g).to(torch.uint8)
    expected_loss = torch.nn.functional.cross_entropy(logits.float(), targets.long(), reduction="none")
    probs = torch.softmax(logits.float(), -1)
    probs[torch.arange(rows), targets.long()] -= 1
    d_logits, d_targets = logits.cuda(), targets.cuda()
    losses = torch.empty(rows, device="cuda")
    grads = torch.empty(rows, 256, device="cuda", dtype=torch.bfloat16)
    scale = 1.0 / rows
    assert lib.tg_ex_cross_entropy(d_logits.data_ptr(), d_targets.data_ptr(), losses.data_ptr(), grads.data_ptr(),
                                   rows, scale, None) == 0
    torch.cuda.synchronize()
    np.testing.assert_allclose(losses.cpu().numpy(), expected_loss.numpy(), rtol=1e-5, atol=1e-5)
    assert max_relative(grads.float().cpu().numpy(), (probs * scale).numpy()) <= 4e-3


@pytest.mark.parametrize("rows,width", [(4096 + 3, 768), (300, 256), (33000, 768), (128, 64)])
def test_head_and_cross_entropy_in_one_kernel(rows, width):
    """The training step's head: logits stay in FP32 inside the kernel (cuda/model.cuh:31-58)."""
    lib = load_library()
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(rows, width, generator=g, device="cuda").bfloat16()
    head = (torch.randn(256, width, generator=g, device="cuda") * (4.0 / width ** 0.5)).bfloat16()
    targets = torch.randint(0, 256, (rows,), generator=g, device="cuda").to(torch.uint8)
    losses = torch.empty(rows, device="cuda")
    grads = torch.empty(rows, 256, device="cuda", dtype=torch.bfloat16)
    scale = 1.0 / rows
    assert lib.tg_ex_head_cross_entropy(x.data_ptr(), head.data_ptr(), targets.data_ptr(), losses.data_ptr(),
                                        grads.data_ptr(), rows, width, scale, None) == 0, lib.tg_error()
    torch.cuda.synchronize()
    logits = x.double() @ head.double().T
    expected = torch.nn.functional.cross_entropy(logits, targets.long(), reduction="none")
    probabilities = torch.softmax(logits, -1)
    probabilities[torch.arange(rows), targets.long()] -= 1
    torch.testing.assert_close(losses.double(), expected, rtol=2e-5, atol=2e-5)
    assert max_relative(grads.float().cpu().numpy(), (probabilities * scale).float().cpu().numpy()) <= 4e-3
    # the loss alone (evaluation), and the same bits on a second call
    again = torch.empty_like(losses)
    assert lib.tg_ex_head_cross_entropy(x.data_ptr(), head.data_ptr(), targets.data_ptr(), again.data_ptr(), None,
                                        rows, width, scale, None) == 0, lib.tg_error()
    torch.cuda.synchronize()
    assert torch.equal(again, losses)


@pytest.mark.parametrize("batch,context,heads,d_head", [(2, 128, 2, 64), (1, 200, 3, 64), (2, 64, 2, 32),
                                                        (2, 1024, 2, 64), (3, 520, 1, 64), (1, 8, 1, 64),
                                                        (2, 40, 2, 64), (1, 65, 1, 64)])
def test_attention_matches_torch(batch, context, heads, d_head):
    lib = load_library()
    width = heads * d_head
    g = torch.Generator().manual_seed(1)
    qkv = torch.randn(batch * context, 3 * width, generator=g).bfloat16()
    dout = torch.randn(batch * context, width, generator=g).bfloat16()
    q, k, v = [t.reshape(batch, context, heads, d_head).transpose(1, 2).float().requires_grad_() for t in qkv.split(width, -1)]
    mask = torch.ones(context, context, dtype=torch.bool).tril()
    scores = (q @ k.transpose(-1, -2) / d_head ** .5).masked_fill(~mask, float("-inf"))
    out = torch.softmax(scores, -1) @ v
    out.backward(dout.reshape(batch, context, heads, d_head).transpose(1, 2).float())
    expected_out = out.detach().transpose(1, 2).reshape(batch * context, width).numpy()
    expected_dqkv = torch.cat([t.grad.transpose(1, 2).reshape(batch * context, width) for t in (q, k, v)], -1).numpy()
    d_qkv, d_dout = qkv.cuda(), dout.cuda()
    d_out = torch.empty(batch * context, width, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(batch * heads * context, device="cuda")
    d_dqkv = torch.empty_like(d_qkv)
    for tensor_cores in ((0, 1) if d_head == 64 else (0,)):
        d_out.zero_()
        lse.zero_()
        assert lib.tg_ex_attention_forward(d_qkv.data_ptr(), d_out.data_ptr(), lse.data_ptr(), batch, context, heads,
                                           d_head, tensor_cores, None) == 0, lib.tg_error()
        torch.cuda.synchronize()
        assert max_relative(d_out.float().cpu().numpy(), expected_out) <= 1e-2, tensor_cores
        expected_lse = torch.logsumexp(scores, -1).detach().reshape(-1).numpy()
        np.testing.assert_allclose(lse.cpu().numpy(), expected_lse, rtol=1e-4, atol=1e-4)
        if tensor_cores and not BACKWARD_ON_TENSOR_CORES:
            continue
        for form in ((1, 2) if tensor_cores else (0,)):  # 2: the single-pass tensor-core kernel
            d_dqkv.zero_()
            assert lib.tg_ex_attention_backward(d_qkv.data_ptr(), d_out.data_ptr(), d_dout.data_ptr(), lse.data_ptr(),
                                                d_dqkv.data_ptr(), batch, context, heads, d_head, form, None) == 0, \
                lib.tg_error()
            torch.cuda.synchronize()
            assert max_relative(d_dqkv.float().cpu().numpy(), expected_dqkv) <= 1e-2, form


@pytest.mark.parametrize("rows,width", [(1000, 768), (515, 256), (300, 1024), (64, 96)])
@pytest.mark.parametrize("kind", [0, 1])
def test_norms_match_torch(rows, width, kind):
    """RMSNorm / LayerNorm forward and backward (with the running residual gradient) as stand-alone
    kernels against FP32 PyTorch: outputs within one BF16 rounding, scale and bias gradients (FP32,
    fixed-order sums over rows) to 1e-4, and the same bits on a second call."""
    from turbogpt_b200.microbench import split_fp32
    lib = load_library()
    g = torch.Generator().manual_seed(3)
    x = (torch.randn(rows, width, generator=g) * 2 + .3).bfloat16()
    dy = torch.randn(rows, width, generator=g).bfloat16()
    residual = torch.randn(rows, width, generator=g).bfloat16()
    scale = 1 + .2 * torch.randn(width, generator=g)
    bias = .1 * torch.randn(width, generator=g)
    xf = x.float().requires_grad_()
    sf, bf = scale.clone().requires_grad_(), bias.clone().requires_grad_()
    if kind == 1:
        expected = torch.nn.functional.layer_norm(xf, (width,), sf, bf, eps=1e-5)
    else:
        expected = torch.nn.functional.rms_norm(xf, (width,), sf, eps=1e-6)
    expected.backward(dy.float())
    d_x, d_dy, d_res = x.cuda(), dy.cuda(), residual.cuda()
    halves = [t.cuda() for t in (*split_fp32(scale), *split_fp32(bias))]
    y = torch.zeros_like(d_x)
    stats = torch.zeros(rows, 2, device="cuda")
    assert lib.tg_ex_norm_forward(kind, d_x.data_ptr(), halves[0].data_ptr(), halves[1].data_ptr(), halves[2].data_ptr(),
                                  halves[3].data_ptr(), y.data_ptr(), stats.data_ptr(), rows, width, None) == 0, lib.tg_error()
    torch.cuda.synchronize()
    assert max_relative(y.float().cpu().numpy(), expected.detach().numpy()) <= 2.0 ** -8
    results = []
    for saved in (stats.data_ptr(), stats.data_ptr(), None):  # twice with the saved statistics, once recomputing them
        dx = torch.zeros_like(d_x)
        dscale, dbias = torch.zeros(width, device="cuda"), torch.zeros(width, device="cuda")
        assert lib.tg_ex_norm_backward(kind, d_x.data_ptr(), d_dy.data_ptr(), halves[0].data_ptr(), halves[1].data_ptr(),
                                       d_res.data_ptr(), saved, dx.data_ptr(), dscale.data_ptr(), dbias.data_ptr(), rows,
                                       width, None) == 0, lib.tg_error()
        torch.cuda.synchronize()
        results.append((dx.float().cpu().numpy(), dscale.cpu().numpy(), dbias.cpu().numpy()))
    recomputed = results.pop()
    assert max_relative(recomputed[0], results[0][0]) <= 2.0 ** -7
    assert max_relative(recomputed[1], results[0][1]) <= 1e-4
    dx, dscale, dbias = results[0]
    expected_dx = residual.float() + xf.grad.bfloat16().float()  # rounded, then added to the residual gradient
    assert max_relative(dx, expected_dx.numpy()) <= 2.0 ** -7
    assert max_relative(dscale, sf.grad.numpy()) <= 1e-4
    if kind == 1:
        assert max_relative(dbias, bf.grad.numpy()) <= 1e-4
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("batch,context,heads", [(700, 1, 1), (304, 64, 2), (301, 65, 2), (160, 129, 2), (61, 333, 4)])
def test_attention_with_four_blocks_per_sm(batch, context, heads):
    """Grids large enough for the one-chain forward kernel, at sequence ends on and off its 64- and 128-row steps."""
    test_attention_matches_torch(batch, context, heads, 64)


def attention_forward(qkv, batch, context, heads):
    lib = load_library()
    out = torch.full((batch * context, heads * 64), float("nan"), device="cuda", dtype=torch.bfloat16)
    lse = torch.full((batch, heads, context), float("nan"), device="cuda")
    assert lib.tg_ex_attention_forward(qkv.data_ptr(), out.data_ptr(), lse.data_ptr(), batch, context, heads, 64, 1, None) == 0, lib.tg_error()
    return out, lse


def attention_backward(qkv, out, dout, lse, batch, context, heads):
    lib, dqkv = load_library(), torch.full_like(qkv, float("nan"))
    assert lib.tg_ex_attention_backward(qkv.data_ptr(), out.data_ptr(), dout.data_ptr(), lse.data_ptr(), dqkv.data_ptr(), batch, context,
                                        heads, 64, 1, None) == 0, lib.tg_error()
    torch.cuda.synchronize()
    assert lib.tg_ex_last_device_error(None) == 0
    return dqkv


@pytest.mark.parametrize("context,heads", [(1, 4), (64, 3), (65, 4), (128, 37), (129, 3), (333, 4), (512, 3), (513, 3), (1000, 2), (1024, 4),
                                           (1025, 2)])
def test_attention_of_small_grids_keeps_the_bits(context, heads):
    """Up to 148 blocks the forward chains have two score buffers, with more one; dQ runs beside dK and dV up to three blocks an SM,
    seven where a sequence has four tiles at most, and context 1024, then before them.  Sequences do not know of one another: the same bits."""
    tiles = -(-context // 128) * heads
    few, some, many = 148 // tiles, 149 // tiles + 2, (7 if context <= 512 else 3) * 148 // tiles + 1
    assert few * tiles <= 148 < some * tiles < 3 * 148 < many * tiles  # `some`: below the one-chain kernel
    g = torch.Generator(device="cuda").manual_seed(context)
    qkv = torch.randn(many * context, heads * 192, generator=g, device="cuda").bfloat16()
    dout = torch.randn(many * context, heads * 64, generator=g, device="cuda").bfloat16()
    for a, b in zip(attention_forward(qkv[:few * context], few, context, heads), attention_forward(qkv[:some * context], some, context, heads)):
        assert torch.isfinite(b).all() and torch.equal(a, b[:len(a)])
    out, lse = attention_forward(qkv, many, context, heads)
    large = attention_backward(qkv, out, dout, lse, many, context, heads)
    assert torch.isfinite(large).all()
    for n in (few, many - 1):
        rows = n * context
        assert torch.equal(attention_backward(qkv[:rows], out[:rows], dout[:rows], lse[:n], n, context, heads), large[:rows])


@pytest.mark.parametrize("batch,context,heads", [(5, 1, 3), (2, 333, 3), (1, 1024, 2), (300, 129, 2), (2, 1100, 3)])
def test_attention_backward_adds_the_products_of_output_and_gradient_in_their_order(batch, context, heads):
    """delta = rowsum(dO * O) is one FP32 accumulator over pairs of products, in dQ's kernel and in dK and dV's, in one launch (the first
    three) and in two.  A row holds 2^34 and, further on, -2^34 among integers up to 6: what precedes the latter is rounded away, what
    follows stays.  Probabilities are 1 and dP 0, every other sum is exact: the gradients are equal."""
    g = torch.Generator(device="cuda").manual_seed(context)
    rows = batch * context
    small = torch.randint(-3, 4, (rows, heads, 32, 2), generator=g, device="cuda").float()
    o, do = small, torch.ones_like(small)
    first = torch.randint(0, 31, (rows, heads, 1), generator=g, device="cuda")
    second = first + 1 + (torch.rand(rows, heads, 1, generator=g, device="cuda") * (31 - first)).long()
    for at, sign in ((first, 1.), (second, -1.)):
        o[..., 0].scatter_(2, at, 2. ** 17)
        do[..., 0].scatter_(2, at, sign * 2. ** 17)
        o[..., 1].scatter_(2, at, 0.)
    pairs = (o.double() * do.double()).sum(-1)
    delta = (pairs * (torch.arange(32, device="cuda") > second)).sum(-1).view(batch, context, heads, 1).transpose(1, 2)
    q, k, v = torch.zeros(3, rows, heads, 64, device="cuda")
    q[..., :32] = torch.randint(-2, 3, (rows, heads, 32), generator=g, device="cuda")  # Q K^T = 0
    k[..., 32:] = torch.randint(-2, 3, (rows, heads, 32), generator=g, device="cuda")
    qkv, lse = torch.stack([q, k, v], 1).bfloat16().view(rows, -1), torch.zeros(batch, heads, context, device="cuda")
    dqkv = attention_backward(qkv, o.bfloat16().view(rows, -1), do.bfloat16().view(rows, -1), lse, batch, context, heads)
    got_q, got_k, _ = dqkv.view(batch, context, 3, heads, 64).permute(2, 0, 3, 1, 4)
    q, k = (t.double().view(batch, context, heads, 64).transpose(1, 2) for t in (q, k))
    assert torch.equal(got_q, (-delta / 8 * k.cumsum(2)).bfloat16())
    assert torch.equal(got_k, (-delta / 8 * q).flip(2).cumsum(2).flip(2).bfloat16())


def test_attention_forward_of_one_buffer_when_the_row_maximum_keeps_growing():
    test_attention_forward_when_the_row_maximum_keeps_growing(30)  # 270 blocks: two chains of one score buffer each


@pytest.mark.parametrize("batch", [100, 2])  # 900 blocks of 128 queries: one chain per block; 18: two chains
def test_attention_forward_when_the_row_maximum_keeps_growing(batch):
    """Scores that climb by more than 2^8 from step to step: the output accumulator is rescaled between products."""
    lib = load_library()
    context, heads = 320, 3
    g = torch.Generator(device="cuda").manual_seed(7)
    qkv = torch.randn(batch * context, 3, heads, 64, generator=g, device="cuda")
    climb = torch.linspace(0, 40, context, device="cuda").repeat(batch)
    qkv[:, 0, :, 0], qkv[:, 1, :, 0] = 64.0, climb[:, None]  # score ~ 8 * climb: up to 320 above the first keys
    qkv = qkv.bfloat16().reshape(batch * context, -1)
    out = torch.empty(batch * context, heads * 64, device="cuda", dtype=torch.bfloat16)
    lse = torch.empty(batch, heads, context, device="cuda")
    assert lib.tg_ex_attention_forward(qkv.data_ptr(), out.data_ptr(), lse.data_ptr(), batch, context, heads, 64, 1,
                                       None) == 0, lib.tg_error()
    torch.cuda.synchronize()
    q, k, v = qkv.reshape(batch, context, 3, heads, 64).permute(2, 0, 3, 1, 4).double()
    scores = (q @ k.transpose(-1, -2) / 8).masked_fill(~torch.ones(context, context, dtype=torch.bool, device="cuda").tril(),
                                                       float("-inf"))
    expected = (torch.softmax(scores, -1) @ v).transpose(1, 2).reshape(batch * context, -1)
    # FP32 scores of ~320 carry 2e-5, their exponentials as much; BF16 probabilities and outputs 2^-8 each
    assert max_relative(out.double().cpu().numpy(), expected.cpu().numpy()) <= 1e-2
    torch.testing.assert_close(lse.double(), torch.logsumexp(scores, -1), rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("rows,width", [(37, 128), (515, 136), (300, 248), (129, 264), (2331, 384), (700, 520),
                                        (260, 1000), (9, 1016)])
@pytest.mark.parametrize("kind", [0, 1])
def test_norms_at_widths_off_the_register_tile(rows, width, kind):
    """Widths that fill the last 256 columns of a row partly: same checks, same bounds."""
    test_norms_match_torch(rows, width, kind)


@pytest.mark.parametrize("rows,width", [(5000, 768), (4801, 776), (5000, 1016), (7103, 1024)])  # up to 768 columns a row's values stay in registers
@pytest.mark.parametrize("kind", [0, 1])
def test_norms_of_several_rows_a_warp(rows, width, kind):
    """More rows than the backward kernel has warps, on both sides of its forms: same checks, same bounds."""
    test_norms_match_torch(rows, width, kind)


@pytest.mark.parametrize("d_head", [64, 32])  # tiles of 64 x 64 positions; a warp per row
@pytest.mark.parametrize("at", [40, 90])      # in the first tile, in the last
def test_cuda_core_attention_keeps_a_later_infinity_out(d_head, at):
    """Causality holds for infinities and NaN too: what precedes (for gradients of keys: follows) one position's infinite
    values has the same bits as without them."""
    lib = load_library()
    batch, context, heads = 2, 100, 2
    g = torch.Generator(device="cuda").manual_seed(3)
    width = heads * d_head

    def run(qkv, dout):
        out = torch.empty_like(dout)
        lse = torch.empty(batch, heads, context, device="cuda")
        dqkv = torch.empty_like(qkv)
        sizes = batch, context, heads, d_head
        assert lib.tg_ex_attention_forward(qkv.data_ptr(), out.data_ptr(), lse.data_ptr(), *sizes, 0, None) == 0, lib.tg_error()
        assert lib.tg_ex_attention_backward(qkv.data_ptr(), out.data_ptr(), dout.data_ptr(), lse.data_ptr(), dqkv.data_ptr(),
                                            *sizes, 0, None) == 0, lib.tg_error()
        torch.cuda.synchronize()
        return out.view(batch, context, -1), lse, dqkv.view(batch, context, 3, -1)

    qkv = torch.randn(batch * context, 3 * width, generator=g, device="cuda").bfloat16()
    dout = torch.randn(batch * context, width, generator=g, device="cuda").bfloat16()
    out, lse, dqkv = run(qkv, dout)
    keys = qkv.clone().view(batch, context, 3, width)
    keys[:, at, 1:] = float("inf")
    out2, lse2, dqkv2 = run(keys.view_as(qkv), dout)
    assert torch.equal(out2[:, :at], out[:, :at]) and torch.equal(lse2[..., :at], lse[..., :at])
    assert torch.equal(dqkv2[:, :at, 0], dqkv[:, :at, 0])
    queries, grown = qkv.clone().view(batch, context, 3, width), dout.clone().view(batch, context, width)
    queries[:, at, 0], grown[:, at] = float("inf"), float("inf")
    _, _, dqkv2 = run(queries.view_as(qkv), grown.view_as(dout))
    assert torch.equal(dqkv2[:, at + 1:, 1:], dqkv[:, at + 1:, 1:])


@pytest.mark.parametrize("rows,width", [(64, 96), (37, 128), (515, 136), (129, 264), (2331, 384), (700, 520), (260, 1000),
                                        (300, 1024), (20, 1032)])
@pytest.mark.parametrize("kind", [0, 1])
def test_norm_statistics_are_kept_at_every_width_that_documents_them(rows, width, kind):
    """Widths 128 to 1024: `stats` receives the row's mean and 1/sigma (FP32 sums: 1e-5 of the value, of sigma for the mean) and
    backward uses them; at other widths it stays untouched.  The array is aligned to its floats only."""
    from turbogpt_b200.microbench import split_fp32
    lib = load_library()
    g = torch.Generator().manual_seed(4)
    x = (torch.randn(rows, width, generator=g) * 2 + .3).bfloat16()
    dy = torch.randn(rows, width, generator=g).bfloat16().cuda()
    halves = [t.cuda() for t in (*split_fp32(1 + .2 * torch.randn(width, generator=g)), *split_fp32(torch.zeros(width)))]
    d_x, y = x.cuda(), torch.empty_like(x, device="cuda")
    stats = torch.full((2 * rows + 1,), float("nan"), device="cuda")[1:]
    assert lib.tg_ex_norm_forward(kind, d_x.data_ptr(), halves[0].data_ptr(), halves[1].data_ptr(), halves[2].data_ptr(),
                                  halves[3].data_ptr(), y.data_ptr(), stats.data_ptr(), rows, width, None) == 0, lib.tg_error()
    torch.cuda.synchronize()
    got = stats.cpu().double().reshape(rows, 2)
    if not 128 <= width <= 1024:
        assert torch.isnan(got).all()
        return
    xd = x.double()
    mean = xd.mean(1) if kind == 1 else torch.zeros(rows, dtype=torch.float64)
    sigma = ((xd - mean[:, None]).square().mean(1) + (1e-5 if kind == 1 else 1e-6)).sqrt()
    assert ((got[:, 0] - mean).abs() <= 1e-5 * sigma).all()
    assert ((got[:, 1] * sigma - 1).abs() <= 1e-5).all()

    def backward(saved):
        dx, dscale, dbias = torch.empty_like(d_x), torch.empty(width, device="cuda"), torch.empty(width, device="cuda")
        assert lib.tg_ex_norm_backward(kind, d_x.data_ptr(), dy.data_ptr(), halves[0].data_ptr(), halves[1].data_ptr(), None,
                                       saved.data_ptr() if saved is not None else None, dx.data_ptr(), dscale.data_ptr(),
                                       dbias.data_ptr(), rows, width, None) == 0, lib.tg_error()
        torch.cuda.synchronize()
        return dx

    assert torch.equal(backward(stats), backward(None))  # recomputed by the same sums
    doubled = torch.empty(2 * rows + 1, device="cuda")[1:].copy_(stats)
    doubled[1::2] *= 2
    assert not torch.equal(backward(doubled), backward(stats))


@pytest.mark.parametrize("sharpness", [1.0, 4.0])  # factor on the queries: flat rows, rows that few keys dominate
def test_one_chain_attention_is_as_exact_as_two(sharpness):
    """The same sequences in a batch of 2 (grid of the two-chain kernel) and of 12 (one chain): BF16 probabilities and outputs
    in both, so the second is no further from 64 bits than the first.  Their rounding errors are independent: over 1.6 M outputs
    their norms agree within 0.2 %."""
    lib = load_library()
    context, heads = 1024, 12
    g = torch.Generator(device="cuda").manual_seed(11)
    qkv = torch.randn(2 * context, 3, heads, 64, generator=g, device="cuda")
    qkv[:, 0] *= sharpness
    qkv = qkv.bfloat16().reshape(2 * context, -1)
    q, k, v = qkv.view(2, context, 3, heads, 64).permute(2, 0, 3, 1, 4).double()
    scores = (q @ k.transpose(-1, -2) / 8).masked_fill(~torch.ones(context, context, dtype=torch.bool, device="cuda").tril(),
                                                       float("-inf"))
    expected = (torch.softmax(scores, -1) @ v).transpose(1, 2).reshape(2 * context, -1)
    errors = []
    for copies in (1, 6):
        packed = qkv.repeat(copies, 1)
        out = torch.empty(copies * 2 * context, heads * 64, device="cuda", dtype=torch.bfloat16)
        lse = torch.empty(copies * 2, heads, context, device="cuda")
        assert lib.tg_ex_attention_forward(packed.data_ptr(), out.data_ptr(), lse.data_ptr(), copies * 2, context, heads, 64, 1,
                                           None) == 0, lib.tg_error()
        torch.cuda.synchronize()
        errors.append(float((out[:2 * context].double() - expected).norm()))
        torch.testing.assert_close(lse[:2].double(), torch.logsumexp(scores, -1), rtol=1e-6, atol=1e-6)
    assert errors[1] <= 1.002 * errors[0]


@pytest.mark.parametrize("a_mn,b_mn", LAYOUTS)
@pytest.mark.parametrize("m,n,k", [(64, 64, 16), (65, 68, 20), (200, 132, 500), (128, 1028, 36), (1540, 1604, 24), (63, 64, 64),
                                   (64, 66, 32), (72, 64, 18)])  # the last three: forms that the vector loads do not take
def test_cuda_core_products_of_both_kernels_agree(a_mn, b_mn, m, n, k):
    """The register-blocked kernel at the edges of its rule and its 64- and 128-wide tiles, rows padded to another stride, against
    64 bits; and against the general kernel, which takes the same operands from an odd element on.  Both add the products in
    ascending k: FP32 sums of k BF16 products, BF16 outputs at most one rounding apart."""
    lib = load_library()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a, b = (torch.randn(rows, k, generator=g, device="cuda").bfloat16() for rows in (m, n))
    expected = a.double() @ b.double().T
    magnitude = a.double().abs() @ b.double().abs().T  # a sum of k terms is off by at most k x 2^-24 of theirs

    def stored(x, transposed, shift):
        x = x.T if transposed else x
        ld = x.shape[1] + 4
        memory = torch.zeros(x.shape[0] * ld + shift, device="cuda", dtype=torch.bfloat16)[shift:]
        rows = memory.view(x.shape[0], ld)
        rows[:, :x.shape[1]] = x
        return memory, (1, ld) if transposed else (ld, 1)

    for out_fp32 in (True, False):
        results = []
        for shift in (0, 1):
            (da, sa), (db, sb) = stored(a, a_mn, shift), stored(b, b_mn, shift)
            c = torch.zeros(m, n, device="cuda", dtype=torch.float32 if out_fp32 else torch.bfloat16)
            assert lib.tg_ex_gemm(da.data_ptr(), *sa, db.data_ptr(), *sb, c.data_ptr(), n, m, n, k, int(out_fp32), 0, None) == 0, \
                lib.tg_error()
            torch.cuda.synchronize()
            bound = k * 2.0 ** -24 * magnitude + (0 if out_fp32 else 2.0 ** -8 * expected.abs())
            assert ((c.double() - expected).abs() <= bound).all(), shift
            results.append(c.double())
        bound = 2 * k * 2.0 ** -24 * magnitude + (0 if out_fp32 else 2.0 ** -7 * expected.abs())
        assert ((results[0] - results[1]).abs() <= bound).all()
