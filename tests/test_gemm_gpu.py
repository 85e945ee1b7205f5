"""tcgen05 GEMM against a plain fp32 PyTorch reference, all four operand layouts, tails, batch, accumulate."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, trans_a, trans_b):
    af = a.float().transpose(-1, -2) if trans_a else a.float()
    bf = b.float().transpose(-1, -2) if trans_b else b.float()
    return af @ bf


def _rand(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * 0.5).to(torch.bfloat16)


@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("mnk", [(128, 256, 64), (256, 512, 256), (384, 320, 192), (200, 136, 72), (1024, 2048, 512)])
def test_gemm_layouts(trans_a, trans_b, mnk):
    from research_b200.ops import native

    M, N, K = mnk
    a = _rand((K, M) if trans_a else (M, K), 1)
    b = _rand((N, K) if trans_b else (K, N), 2)
    out = native.gemm(a, b, trans_a=trans_a, trans_b=trans_b)
    native.check_status()
    ref = _ref(a, b, trans_a, trans_b)
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, (err, scale)


@pytest.mark.parametrize("bn", [128, 256])
def test_gemm_fp32_out_and_accumulate(bn):
    from research_b200.ops import native

    M, N, K = 512, 768, 320
    a, b = _rand((M, K), 3), _rand((N, K), 4)
    out = native.gemm(a, b, out_dtype=torch.float32, bn=bn)
    ref = _ref(a, b, False, True)
    assert (out - ref).abs().max().item() <= 2e-3 * ref.abs().max().item() + 1e-3
    native.gemm(a, b, out=out, accumulate=True, bn=bn)
    native.check_status()
    assert (out - 2 * ref).abs().max().item() <= 4e-3 * ref.abs().max().item() + 2e-3


def test_gemm_batched_and_strided_rows():
    from research_b200.ops import native

    B, M, N, K = 3, 256, 384, 128
    a, b = _rand((B, M, K), 5), _rand((B, N, K), 6)
    out = native.gemm(a, b)
    ref = _ref(a, b, False, True)
    assert (out.float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item() + 1e-2
    wide = _rand((M, 2 * K), 7)
    a2 = wide[:, :K]  # row stride 2K
    out2 = native.gemm(a2, b[0])
    native.check_status()
    ref2 = _ref(a2, b[0], False, True)
    assert (out2.float() - ref2).abs().max().item() <= 1e-2 * ref2.abs().max().item() + 1e-2


def test_gemm_large_matches_and_is_timed():
    from research_b200.ops import native

    M = N = K = 4096
    a, b = _rand((M, K), 8), _rand((N, K), 9)
    out = native.gemm(a, b)
    ref = (a @ b.t()).float()
    assert (out.float() - ref).abs().max().item() <= 2e-2 * ref.abs().max().item()
    for _ in range(3):
        native.gemm(a, b, out=out)
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(10):
        native.gemm(a, b, out=out)
    e.record()
    torch.cuda.synchronize()
    native.check_status()
    tflops = 10 * 2 * M * N * K / (s.elapsed_time(e) * 1e-3) / 1e12
    print(f"gemm 4096^3: {tflops:.1f} TFLOP/s")
    assert tflops > 50


def test_skinny_splitk_gemm_matches_reference():
    from research_b200.ops import native

    torch.manual_seed(0)
    # nothing is kept between calls: large after small and back again, each shape as often as it comes
    for rows, n, k in ((32, 2048, 2048), (32, 2048, 5632), (7, 11264, 2048), (64, 4096, 2048), (3, 512, 256),
                       (64, 11264, 2048), (32, 2048, 2048)):
        a = (torch.randn(rows, k, device="cuda") * 0.5).bfloat16()
        b = (torch.randn(n, k, device="cuda") * 0.05).bfloat16()
        ref = a.float() @ b.float().t()
        for fused in (False, True):       # a switch of earlier callers: accepted, the result is the same
            y = native.gemm_skinny(a, b, fused_finish=fused)
            native.check_status()
            assert y.shape == (rows, n) and y.dtype == torch.bfloat16
            assert torch.allclose(y.float(), ref, atol=3e-2, rtol=3e-2), (rows, n, k, fused, (y.float() - ref).abs().max().item())
    assert native.splitk_factor(2048, 2048) > 1


def test_weight_gradient_split_k_accumulates_like_one_pass():
    from research_b200.ops import native

    torch.manual_seed(0)
    for tokens, m, n in ((8192, 2048, 2048), (4096, 2048, 5632), (2048, 512, 256)):
        dy = (torch.randn(tokens, m, device="cuda") * 0.1).bfloat16()
        x = (torch.randn(tokens, n, device="cuda") * 0.5).bfloat16()
        grad = torch.full((m, n), 0.25, dtype=torch.float32, device="cuda")
        native.gemm_wgrad(dy, x, grad)
        native.check_status()
        ref = 0.25 + dy.float().t() @ x.float()
        assert (grad - ref).abs().max().item() <= 2e-3 * ref.abs().max().item() + 1e-3
    assert native.wave_splits(2048, 2048, 32768) > 1


# tokens that are no multiple of a 64-element block of K and fewer than two slices: one pass, the same bits every time
@pytest.mark.parametrize("tokens", [1, 63, 130, 777, 1024, 1984, 2999])
@pytest.mark.parametrize("m,n", [(128, 256), (1024, 512), (520, 264)])
def test_weight_gradient_in_one_pass(tokens, m, n):
    from research_b200.ops import native

    torch.manual_seed(1)
    dy = (torch.randn(tokens, m, device="cuda") * 0.1).bfloat16()
    x = (torch.randn(tokens, n, device="cuda") * 0.5).bfloat16()
    grads = []
    for _ in range(20):
        grads.append(torch.full((m, n), 0.25, dtype=torch.float32, device="cuda"))
        native.gemm_wgrad(dy, x, grads[-1])
    native.check_status()
    assert all(torch.equal(grads[0], g) for g in grads)
    ref = 0.25 + dy.double().t() @ x.double()
    # exact products, fp32 sums of at most 2999 of them in any order: 2999 * 2^-24 of the sum of magnitudes, far from reached
    assert (grads[0].double() - ref).abs().max() <= 2.0 ** -18 * (dy.double().abs().t() @ x.double().abs()).max() + 2.0 ** -24


# sizes around the edges of a 128-row block and of the narrow and the wide tile, odd numbers of blocks, both operand
# layouts; batches that make the launcher take either tile width
@pytest.mark.parametrize("d", [8, 64, 128, 136, 256, 384, 520, 1024, 1160])
@pytest.mark.parametrize("K", [8, 200, 512])
@pytest.mark.parametrize("batch", [1, 3, 20])
def test_gram_is_symmetric_and_exact(d, K, batch):
    from research_b200.ops import native

    torch.manual_seed(d + K)
    for transposed in (False, True):
        x = (torch.randn((batch, K, d) if transposed else (batch, d, K), device="cuda") * 0.1).bfloat16()
        g = native.gram(x, transposed=transposed)
        xd = x.double().transpose(1, 2) if transposed else x.double()
        ref = xd @ xd.transpose(1, 2)
        assert torch.equal(g, g.transpose(1, 2))
        assert (g.double() - ref).norm() <= 2.0 ** -8 * ref.norm()       # one rounding to bf16: 2^-8 of a value at most
    q = native.gram(g, alpha=2.0, beta=-4.75, gamma=3.5)
    gd = g.double()
    ref = 2.0 * gd @ gd - 4.75 * gd + 3.5 * torch.eye(d, device="cuda", dtype=torch.float64)
    native.check_status()
    assert torch.equal(q, q.transpose(1, 2))
    assert (q.double() - ref).norm() <= 2.0 ** -8 * ref.norm()
    with pytest.raises(native.KernelError):
        native.gram(x[:, :, :4] if d != 4 else x)


# every form of stack that plain products take: rows that are no multiple of 8 where there are more rows than columns,
# rows and matrices at a distance, a single matrix
@pytest.mark.parametrize("shape", [(2, 1001, 512), (3, 130, 64), (2, 256, 520), (1, 70, 64), (300, 136), (136, 264)])
@pytest.mark.parametrize("apart", [0, 8])
def test_newton_schulz_takes_every_stack_that_products_take(shape, apart):
    from research_b200.ops import native
    from research_b200.optim import orthogonalize as orth

    torch.manual_seed(shape[-1])
    x = torch.randn(shape, device="cuda")
    wide = torch.zeros(*shape[:-2], shape[-2] + apart, shape[-1] + apart, device="cuda", dtype=torch.bfloat16)
    stack = wide[..., :shape[-2], :shape[-1]].copy_(x / torch.linalg.matrix_norm(x, keepdim=True))
    got = orth.newton_schulz_stack_(stack)
    native.check_status()
    ref = stack.double()
    if shape[-2] > shape[-1]:
        ref = ref.transpose(-1, -2)
    for _ in range(orth.MUON_NS_STEPS):
        a, b, c = orth.MUON_NS_COEFFICIENTS
        g = ref @ ref.transpose(-1, -2)
        ref = a * ref + (b * g + c * g @ g) @ ref
    ref = ref.transpose(-1, -2) if shape[-2] > shape[-1] else ref
    # five steps, each with three roundings to bf16 that the next step's slope (up to 3.4445) amplifies
    assert got.shape == stack.shape and (got.double() - ref).norm() <= 5 * 3 * 2.0 ** -8 * ref.norm()


# rows on both sides of each tile width, weight rows and K that are no multiple of a tile or of the slices, one slice to
# eight, output widths that are no multiple of four
@pytest.mark.parametrize("rows", [1, 16, 17, 33, 64, 100, 128])
@pytest.mark.parametrize("n,k", [(8, 64), (130, 128), (2048, 2048), (1000, 1856), (11264, 512), (2046, 320), (333, 704)])
def test_skinny_products(rows, n, k):
    from research_b200.ops import native

    torch.manual_seed(rows + n)
    x = torch.randn(rows, k + 8, device="cuda").bfloat16()[:, :k]
    w = (torch.randn(n, k, device="cuda") * 0.05).bfloat16()
    y = native.gemm_skinny(x, w)
    again = native.gemm_skinny(x, w)
    native.check_status()
    ref = x.double() @ w.double().t()
    assert y.shape == (rows, n) and torch.equal(y, again)
    assert (y.double() - ref).norm() <= 2.0 ** -8 * ref.norm()           # one rounding to bf16
    lib = native.load()
    for slices in (1, 2, 4, 8):                                          # more slices than blocks of K leave some empty
        out = torch.full((rows, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        assert lib.b200_gemm_skinny(x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, n, k, slices, x.stride(0), k, n,
                                    native.status_word(x.device).data_ptr(), native._stream()) == 0
        assert (out.double() - ref).norm() <= 2.0 ** -8 * ref.norm()
    native.check_status()


@pytest.mark.parametrize("rows,n,k", [(1, 128, 2048), (32, 2048, 4096), (64, 512, 512)])
def test_skinny_product_with_weights_that_its_predecessor_writes(rows, n, k):
    """W straight out of another such product, and an fp32 parameter that is cast on every call: bit for bit what it
    is with the device idle before each product."""

    from research_b200.ops import functional as Fn
    from research_b200.ops import native

    torch.manual_seed(k)
    x = torch.randn(rows, k, device="cuda").bfloat16()
    a = torch.randn(128, 512, device="cuda").bfloat16()
    b = [(torch.randn(k, 512, device="cuda") * 0.05).bfloat16() for _ in range(4)]
    start = torch.randn(n, k, device="cuda") * 0.05
    p = torch.nn.Parameter(start.clone())
    runs = []
    with torch.no_grad():
        for idle in (True, False):
            p.copy_(start)
            got = []
            for i in range(24):
                w = native.gemm_skinny(a, b[i % 4])
                if idle:
                    torch.cuda.synchronize()
                got.append(native.gemm_skinny(x, w))
                p.mul_(-1.25 if i % 2 else 0.8)
                if idle:
                    torch.cuda.synchronize()
                got.append(Fn.linear(x, p))
            runs.append(got)
    native.check_status()
    assert all(torch.equal(u, v) for u, v in zip(*runs))


# the product on CTA pairs (bn=512) against 64 bits: edges of its 256 x 256 tile, a second CTA without rows or columns,
# K shorter than a block and longer than the ring, more tiles than pairs, batches, accumulation
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (128, 256, 64), (129 * 8, 264, 72), (256, 136, 448), (520, 1000, 1000),
                                   (2304, 2560, 128)])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
def test_products_on_cta_pairs(M, N, K, ta, tb):
    from research_b200.ops import native

    torch.manual_seed(M + K)
    for batch in (1, 3):
        a = torch.randn((batch, K, M) if ta else (batch, M, K), device="cuda").bfloat16()
        b = torch.randn((batch, N, K) if tb else (batch, K, N), device="cuda").bfloat16()
        ad, bd = a.double(), b.double()
        ref = (ad.transpose(1, 2) if ta else ad) @ (bd.transpose(1, 2) if tb else bd)
        size = (ad.abs().transpose(1, 2) if ta else ad.abs()) @ (bd.abs().transpose(1, 2) if tb else bd.abs())
        y = native.gemm(a, b, trans_a=ta, trans_b=tb, bn=512)
        assert (y.double() - ref).norm() <= 2.0 ** -8 * ref.norm()       # one rounding to bf16
        acc = torch.full((batch, M, N), 0.5, device="cuda")
        native.gemm(a, b, trans_a=ta, trans_b=tb, out=acc, accumulate=True, bn=512)
        native.check_status()
        # fp32 sums of K exact products: K * 2^-24 of the sum of magnitudes bounds any order
        assert (acc.double() - ref - 0.5).abs().max() <= K * 2.0 ** -24 * (size.max() + 1)


# long enough for CTA pairs: contractions of uneven length, an empty one among them, with an output that has no whole
# last tile; and K slices that pairs add into one output
@pytest.mark.parametrize("m,n", [(2048, 2048), (2040, 1544)])
def test_pair_products_with_ranges_of_k(m, n):
    from research_b200.ops import native

    torch.manual_seed(3)
    ranges = [0, 4096, 4096, 4160, 8192, 12288]
    a = (torch.randn(ranges[-1], m, device="cuda") * 0.1).bfloat16()
    b = (torch.randn(ranges[-1], n, device="cuda") * 0.5).bfloat16()
    assert ranges[-1] * m * n >= 2.5e10                      # the launcher's rule for pairs
    out = torch.full((len(ranges) - 1, m, n), 0.25, device="cuda")
    bounds = torch.tensor(list(zip(ranges[:-1], ranges[1:])), dtype=torch.int32, device="cuda")
    rc = native.load().b200_gemm_bf16_grouped_k(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, ranges[-1], len(ranges) - 1, m, n, n, m * n, 1, 1,
        bounds.data_ptr(), native.status_word().data_ptr(), native._stream())
    assert rc == 0
    native.check_status()
    for i, (lo, hi) in enumerate(zip(ranges[:-1], ranges[1:])):
        ad, bd = a[lo:hi].double(), b[lo:hi].double()
        # exact products, fp32 sums of at most 4096 of them: the same bound as for one pass over 2999 tokens
        assert (out[i].double() - 0.25 - ad.T @ bd).abs().max() <= 2.0 ** -18 * (ad.abs().T @ bd.abs()).max() + 2.0 ** -24, i


def test_pair_products_with_slices_of_k():
    from research_b200.ops import native

    torch.manual_seed(4)
    k, m, n = 4096, 2048, 5632
    assert native.wave_splits(m, n, k) > 1 and k * m * n >= 2.5e10
    dy, x = (torch.randn(k, m, device="cuda") * 0.1).bfloat16(), (torch.randn(k, n, device="cuda") * 0.5).bfloat16()
    grad = torch.full((m, n), 0.25, device="cuda")
    native.gemm_wgrad(dy, x, grad)
    native.check_status()
    ref, size = dy.double().T @ x.double(), dy.double().abs().T @ x.double().abs()
    assert (grad.double() - 0.25 - ref).abs().max() <= 2.0 ** -18 * size.max() + 2.0 ** -24


def _in_new_thread(fn):
    import threading

    got = []

    def work():
        try:
            got.append(fn())
        except Exception as e:                      # noqa: BLE001 - handed to the test
            got.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    return got[0]


@pytest.mark.parametrize("product", ["gemm", "skinny", "attention"])
def test_first_cuda_work_of_a_thread_can_be_a_product(product):
    """A thread without a current CUDA context, whose first work encodes 3-, 2- and 4-dimensional tensor maps."""

    from research_b200.ops import native

    a, b = _rand((256, 256), 1), _rand((256, 256), 2)
    q = _rand((1, 256, 2, 64), 3)
    run = {"gemm": lambda: native.gemm(a, b), "skinny": lambda: native.gemm_skinny(a[:64], b),
           "attention": lambda: native.attn_fwd(q, q, q)[0]}[product]
    want = run()
    got = _in_new_thread(run)
    torch.cuda.synchronize()
    native.check_status()
    assert torch.is_tensor(got), got
    assert torch.equal(got, want)


def test_first_backward_of_a_process_can_start_with_a_product():
    import subprocess
    import sys
    from pathlib import Path

    code = ("import torch\n"
            "from research_b200.ops import functional as Fn, native\n"
            "x = torch.randn(256, 256, device='cuda').bfloat16().requires_grad_(True)\n"
            "w = torch.nn.Parameter(torch.randn(512, 256, device='cuda').bfloat16())\n"
            "w.main_grad = torch.zeros(512, 256, device='cuda')\n"
            "g = torch.ones(256, 512, device='cuda').bfloat16()\n"
            "(dx,) = torch.autograd.grad([Fn.linear(x, w)], [x], [g])\n"
            "native.check_status()\n"
            "assert torch.allclose(dx.float(), w.float().sum(0).expand(256, 256), rtol=2e-2, atol=0.2)\n")
    done = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, capture_output=True,
                          text=True, timeout=300)
    assert done.returncode == 0, done.stderr


def test_first_products_of_a_process_from_several_threads_at_once():
    import subprocess
    import sys
    from pathlib import Path

    code = ("import threading, torch\n"
            "from research_b200.ops import native\n"
            "native.load(), native.status_word()\n"
            "a = torch.ones(128, 128, device='cuda', dtype=torch.bfloat16)\n"
            "gate, got = threading.Barrier(16), []\n"
            "def work():\n"
            "    gate.wait()\n"
            "    try: got.append(native.gemm(a, a))\n"
            "    except Exception as e: got.append(e)\n"
            "threads = [threading.Thread(target=work) for _ in range(16)]\n"
            "[t.start() for t in threads], [t.join() for t in threads]\n"
            "torch.cuda.synchronize(), native.check_status()\n"
            "assert all(torch.is_tensor(g) and (g == 128).all() for g in got), got\n")
    for _ in range(3):
        done = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, capture_output=True,
                              text=True, timeout=300)
        assert done.returncode == 0, done.stderr
