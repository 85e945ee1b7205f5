"""Bandwidth-bound kernels against fp32 PyTorch restatements of the same math."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("H", [128, 2048, 4096, 1000])
@pytest.mark.parametrize("rows", [77, 1500])   # one block per row below 512 rows, one warp per row above
def test_rmsnorm_fwd_bwd(H, rows):
    from research_b200.ops import native

    eps = 1e-6
    x, delta, dy = _bf((rows, H), 1), _bf((rows, H), 2), _bf((rows, H), 3)
    w = torch.rand(H, device="cuda") + 0.5
    y, rstd, res = native.rmsnorm_fwd(x, w, eps, delta)
    resf = (x.float() + delta.float()).to(torch.bfloat16).float()
    ref = resf * torch.rsqrt(resf.pow(2).mean(-1, keepdim=True) + eps) * w
    assert torch.allclose(res.float(), resf, atol=1e-2, rtol=1e-2)
    assert torch.allclose(y.float(), ref, atol=3e-2, rtol=2e-2)
    xr = res.float().requires_grad_(True)
    wr = w.clone().requires_grad_(True)
    yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + eps) * wr
    yr.backward(dy.float())
    dw = torch.zeros(H, device="cuda")
    dx = native.rmsnorm_bwd(res, w, rstd, dy, dw)
    assert torch.allclose(dx.float(), xr.grad, atol=3e-2, rtol=3e-2)
    assert torch.allclose(dw, wr.grad, atol=5e-2, rtol=2e-2)


@pytest.mark.parametrize("H", [128, 768, 2048, 4096])
@pytest.mark.parametrize("rows", [3, 600])
def test_norm_scales_are_read_in_the_precision_they_are_held_in(H, rows):
    """The parameter store holds norm scales as bf16 compute copies: the kernels give bit for bit what they give for
    the same values in fp32, for RMSNorm and for the QK-norm, forward and backward."""

    from research_b200.ops import native

    x, dy = _bf((rows, H), 21), _bf((rows, H), 22)
    wb = (torch.rand(H, device="cuda") + 0.5).to(torch.bfloat16)
    got = []
    for w in (wb, wb.float()):
        y, rstd, _ = native.rmsnorm_fwd(x, w, 1e-6)
        out = torch.empty_like(x)
        r = native.qknorm_rope_fwd_qk(x, out, w[:64], w[64:128], torch.arange(rows, device="cuda", dtype=torch.int32), 1,
                                      1, 64, 1e-6, 10000.0, True)
        din, dq, dk = torch.zeros_like(x), torch.zeros(64, device="cuda"), torch.zeros(64, device="cuda")
        native.qknorm_rope_bwd_qk(x, dy, din, w[:64], w[64:128], torch.arange(rows, device="cuda", dtype=torch.int32),
                                  r, dq, dk, 1, 1, 64, 10000.0, True)
        dx = native.rmsnorm_bwd(x, w, rstd, dy, torch.zeros(H, device="cuda"))
        got.append((y, out[:, :128], din[:, :128], dx))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    with pytest.raises(native.KernelError):
        native.rmsnorm_fwd(x, wb.half(), 1e-6)


def _off(got, ref):
    return float((got.detach().double() - ref.detach().double()).norm() / ref.detach().double().norm())


# widths on each side of the kernel's choices of columns per thread (2304, 2816 and 3840 are multiples of 256 that take a
# warp per row), rows around a block's group of rows
@pytest.mark.parametrize("H", [256, 512, 768, 2048, 2304, 2560, 2816, 3840, 4096, 5632, 8192, 8200])
@pytest.mark.parametrize("rows", [1, 5, 1203])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_bwd_widths(H, rows, with_res):
    from research_b200.ops import native

    x, dy = _bf((rows, H), 31), _bf((rows, H), 32)
    dres = _bf((rows, H), 33) if with_res else None
    w = torch.rand(H, device="cuda") + 0.5
    _, rstd, _ = native.rmsnorm_fwd(x, w, 1e-6)
    xr, wr = x.double().requires_grad_(True), w.double().requires_grad_(True)
    (xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr).backward(dy.double())
    dw = torch.ones(H, device="cuda")                                   # accumulated into
    dx = native.rmsnorm_bwd(x, w, rstd, dy, dw, dres)
    # one rounding to bf16 (2^-8 of each value at most); fp32 sums of at most 1203 terms (2^-24 each) on top of the 1
    assert _off(dx, xr.grad + (0 if dres is None else dres.double())) < 2.0 ** -8
    assert _off(dw, wr.grad + 1) < 1e-5


# a weight gradient that starts anywhere in an arena: the same values, by the same kernel
@pytest.mark.parametrize("H", [256, 512, 1024, 2048, 4096, 8192])
def test_rmsnorm_bwd_into_an_unaligned_gradient(H):
    from research_b200.ops import native

    rows = 2 ** 25 // H
    x, dy, w = _bf((rows, H), 31), _bf((rows, H), 32), torch.rand(H, device="cuda") + 0.5
    _, rstd, _ = native.rmsnorm_fwd(x, w, 1e-6)
    arena = torch.zeros(H + 8, device="cuda")

    def run(off):
        return native.rmsnorm_bwd(x, w, rstd, dy, arena[off:off + H])

    def time_us(off):
        best = float("inf")
        for _ in range(5):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record()
            for _ in range(10):
                run(off)
            e.record()
            torch.cuda.synchronize()
            best = min(best, s.elapsed_time(e) * 100)
        return best

    want_dx, want = run(0), arena[:H].clone()
    for off in (1, 2, 3):
        arena.zero_()
        assert torch.equal(run(off), want_dx)
        # fp32 partial sums of at most 2368 blocks in arrival order
        assert _off(arena[off:off + H], want) < 1e-4 and not arena[:off].any() and not arena[off + H:].any()
    # the kernel that walks rows with a warp each takes 1.3 (256 columns) to 3.3 times as long
    slow, fast = time_us(1), time_us(0)
    assert slow < 1.2 * fast, (slow, fast)


# odd head counts, tokens on both sides of the rule that deals a token's heads to several warps (4736 tokens)
@pytest.mark.parametrize("T,hq,hkv,D", [(1, 1, 1, 128), (33, 3, 1, 64), (700, 5, 3, 128), (700, 7, 1, 96),
                                        (4735, 2, 1, 64), (4740, 3, 2, 128), (9, 2, 2, 256), (50, 4, 4, 8)])
def test_qknorm_rope_shapes(T, hq, hkv, D):
    from research_b200.ops import native

    buf, dout = _bf((T, (hq + 2 * hkv) * D), 41), _bf((T, (hq + hkv) * D), 42)
    pos = torch.arange(T, device="cuda", dtype=torch.int32) % 251
    wq, wk = torch.rand(D, device="cuda") + 0.5, torch.rand(D, device="cuda") + 0.5
    out = torch.zeros(T, (hq + hkv) * D, dtype=torch.bfloat16, device="cuda")
    r = native.qknorm_rope_fwd_qk(buf, out, wq, wk, pos, hq, hkv, D, 1e-6, 10000.0, True)
    x = buf[:, :(hq + hkv) * D].double().view(T, hq + hkv, D).requires_grad_(True)
    ws = [wq.double().requires_grad_(True), wk.double().requires_grad_(True)]
    scale = torch.cat([ws[0].expand(hq, D), ws[1].expand(hkv, D)])
    ref = _rope_ref(x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * scale, pos.double(), 10000.0)
    grads = torch.autograd.grad([ref], [x] + ws, [dout.double().view(T, hq + hkv, D)])
    din = torch.zeros_like(buf)
    dq, dk = torch.zeros(D, device="cuda"), torch.zeros(D, device="cuda")
    native.qknorm_rope_bwd_qk(buf, dout, din, wq, wk, pos, r, dq, dk, hq, hkv, D, 10000.0, True)
    same = dout.clone()
    native.qknorm_rope_bwd_qk(buf, same, same, wq, wk, pos, r, torch.zeros_like(dq), torch.zeros_like(dk), hq, hkv, D,
                              10000.0, True)
    # one rounding to bf16; the angle is formed in fp32: 251 * 2^-24 = 1.5e-5
    assert _off(out.view(T, hq + hkv, D), ref) < 2.0 ** -8
    assert _off(din[:, :(hq + hkv) * D].view(T, hq + hkv, D), grads[0]) < 2.0 ** -8
    assert _off(dq, grads[1]) < 1e-4 and _off(dk, grads[2]) < 1e-4
    assert torch.equal(same, din[:, :(hq + hkv) * D]) and not din[:, (hq + hkv) * D:].any()


def _rope_ref(x, pos, theta):
    D = x.shape[-1]
    inv = theta ** (-torch.arange(0, D, 2, device=x.device, dtype=torch.float32) / D)
    ang = pos.float()[:, None, None] * inv
    c, s = ang.cos(), ang.sin()
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, a * s + b * c], dim=-1).flatten(-2)


@pytest.mark.parametrize("D", [32, 64, 128])
def test_qknorm_rope(D):
    from research_b200.ops import native

    T, heads, theta, eps = 50, 6, 10000.0, 1e-6
    stride = heads * D + 64
    buf = _bf((T, stride), 4)
    pos = torch.arange(T, device="cuda", dtype=torch.int32) * 3
    w = torch.rand(D, device="cuda") + 0.5
    out = torch.zeros(T, heads * D, dtype=torch.bfloat16, device="cuda")
    rstd = native.qknorm_rope_fwd(buf, out, w, pos, heads, D, eps, theta, True)
    xin = buf[:, : heads * D].float().view(T, heads, D).requires_grad_(True)
    wr = w.clone().requires_grad_(True)
    xn = xin * torch.rsqrt(xin.pow(2).mean(-1, keepdim=True) + eps) * wr
    ref = _rope_ref(xn, pos, theta)
    assert torch.allclose(out.float().view(T, heads, D), ref, atol=3e-2, rtol=3e-2)
    dout = _bf((T, heads * D), 5)
    ref.backward(dout.float().view(T, heads, D))
    din = torch.zeros(T, heads * D, dtype=torch.bfloat16, device="cuda")
    dw = torch.zeros(D, device="cuda")
    native.qknorm_rope_bwd(buf, dout, din, w, pos, rstd, dw, heads, D, theta, True)
    assert torch.allclose(din.float().view(T, heads, D), xin.grad, atol=4e-2, rtol=4e-2)
    assert torch.allclose(dw, wr.grad, atol=0.15, rtol=3e-2)


@pytest.mark.parametrize("D", [64, 128])
def test_qknorm_rope_packed_qk_matches_two_single_launches(D):
    """Query and key heads in one launch (separate norm weights and weight gradients) against one launch each."""

    from research_b200.ops import native

    T, hq, hkv, theta, eps = 70, 4, 2, 10000.0, 1e-6
    width = (hq + 2 * hkv) * D
    buf = _bf((T, width), 11)
    pos = torch.arange(T, device="cuda", dtype=torch.int32) * 5
    wq, wk = torch.rand(D, device="cuda") + 0.5, torch.rand(D, device="cuda") + 0.5
    dout = _bf((T, (hq + hkv) * D), 12)
    out_a = torch.zeros(T, (hq + hkv) * D, dtype=torch.bfloat16, device="cuda")
    out_b = torch.zeros_like(out_a)
    r = native.qknorm_rope_fwd_qk(buf, out_a, wq, wk, pos, hq, hkv, D, eps, theta, True)
    rq = native.qknorm_rope_fwd(buf, out_b, wq, pos, hq, D, eps, theta, True)
    rk = native.qknorm_rope_fwd(buf[:, hq * D:], out_b[:, hq * D:], wk, pos, hkv, D, eps, theta, True)
    assert torch.equal(out_a, out_b)
    assert torch.equal(r.view(T, hq + hkv)[:, :hq].reshape(-1), rq)
    assert torch.equal(r.view(T, hq + hkv)[:, hq:].reshape(-1), rk)
    din_a = torch.zeros(T, width, dtype=torch.bfloat16, device="cuda")
    din_b = torch.zeros_like(din_a)
    dwq_a, dwk_a = torch.zeros(D, device="cuda"), torch.zeros(D, device="cuda")
    dwq_b, dwk_b = torch.zeros(D, device="cuda"), torch.zeros(D, device="cuda")
    native.qknorm_rope_bwd_qk(buf, dout, din_a, wq, wk, pos, r, dwq_a, dwk_a, hq, hkv, D, theta, True)
    native.qknorm_rope_bwd(buf, dout, din_b, wq, pos, rq, dwq_b, hq, D, theta, True)
    native.qknorm_rope_bwd(buf[:, hq * D:], dout[:, hq * D:], din_b[:, hq * D:], wk, pos, rk, dwk_b, hkv, D, theta, True)
    assert torch.equal(din_a, din_b)
    assert torch.allclose(dwq_a, dwq_b, atol=1e-3, rtol=1e-4) and torch.allclose(dwk_a, dwk_b, atol=1e-3, rtol=1e-4)
    # without norm weights (RoPE only)
    out_c = torch.zeros_like(out_a)
    assert native.qknorm_rope_fwd_qk(buf, out_c, None, None, pos, hq, hkv, D, eps, theta, True) is None
    out_d = torch.zeros_like(out_a)
    native.qknorm_rope_fwd(buf, out_d, None, pos, hq + hkv, D, eps, theta, True)
    assert torch.equal(out_c, out_d)
    native.check_status()


def test_swiglu_and_gate():
    from research_b200.ops import native

    rows, inter = 33, 256
    gu, dh = _bf((rows, 2 * inter), 6), _bf((rows, inter), 7)
    h = native.swiglu_fwd(gu)
    g = gu[:, :inter].float().requires_grad_(True)
    u = gu[:, inter:].float().requires_grad_(True)
    ref = torch.nn.functional.silu(g) * u
    assert torch.allclose(h.float(), ref, atol=2e-2, rtol=2e-2)
    ref.backward(dh.float())
    dgu = native.swiglu_bwd(gu, dh)
    assert torch.allclose(dgu[:, :inter].float(), g.grad, atol=3e-2, rtol=3e-2)
    assert torch.allclose(dgu[:, inter:].float(), u.grad, atol=3e-2, rtol=3e-2)
    a, gate, dout = _bf((rows, inter), 8), _bf((rows, inter), 9), _bf((rows, inter), 10)
    out = native.sigmoid_gate_fwd(a, gate)
    assert torch.allclose(out.float(), a.float() * torch.sigmoid(gate.float()), atol=2e-2, rtol=2e-2)
    da, dg = native.sigmoid_gate_bwd(a, gate, dout)
    sg = torch.sigmoid(gate.float())
    assert torch.allclose(da.float(), dout.float() * sg, atol=2e-2, rtol=2e-2)
    assert torch.allclose(dg.float(), dout.float() * a.float() * sg * (1 - sg), atol=2e-2, rtol=3e-2)


def test_embedding_and_ce():
    from research_b200.ops import native

    V, H, T = 1000, 64, 40
    table = _bf((V, H), 11)
    ids = torch.randint(0, V, (T,), device="cuda", dtype=torch.int32)
    out = native.embedding_fwd(ids, table, 2.0)
    assert torch.allclose(out.float(), table[ids.long()].float() * 2.0, atol=1e-2, rtol=1e-2)
    dtable = torch.zeros(V, H, device="cuda")
    native.embedding_bwd(ids, out, dtable, 1.0)
    ref = torch.zeros(V, H, device="cuda").index_add_(0, ids.long(), out.float())
    assert torch.allclose(dtable, ref, atol=1e-3, rtol=1e-3)


@pytest.mark.parametrize("V2,ld", [(50304, 50304), (1000, 1000), (32768, 32776), (1004, 1008), (128256, 128256)])
def test_cross_entropy_rows_staged_in_shared_memory_and_the_three_pass_form(V2, ld):
    """Rows of at most 200 KB with V % 8 == 0 take the kernel that stages the row in shared memory (one bulk copy in,
    one out); the others the three-pass kernel.  Both against the fp32 autograd oracle, padded row stride included."""

    from research_b200.ops import native

    T = 24
    logits = _bf((T, ld), 12, 2.0)[:, :V2]
    tgt = torch.randint(0, V2, (T,), device="cuda", dtype=torch.int32)
    mask = (torch.rand(T, device="cuda") > 0.2).to(torch.uint8)
    zw, gs = 1e-4, 1.0 / float(mask.sum().item())
    lf = logits.float().requires_grad_(True)
    lse = torch.logsumexp(lf, -1)
    ce = (lse - lf.gather(1, tgt.long()[:, None])[:, 0]) * mask
    obj = (ce.sum() + zw * (lse.pow(2) * mask).sum()) * gs
    obj.backward()
    loss, z, lse_k = native.ce_fwd_bwd(logits, tgt, mask, gs, zw)
    assert torch.allclose(loss, ce.detach(), atol=2e-3, rtol=1e-3)
    assert torch.allclose(z, (lse.pow(2) * mask).detach(), atol=1e-2, rtol=1e-3)
    assert torch.allclose(logits.float(), lf.grad, atol=2e-4, rtol=5e-2)
    assert torch.allclose(lse_k, (lse * mask).detach(), atol=2e-3, rtol=1e-3)
    assert not logits[mask == 0].any()
    native.check_status()


@pytest.mark.parametrize("n,gdtype", [(100_003, torch.bfloat16), (100_000, torch.bfloat16), (65_536, torch.float32)])
def test_adamw_sumsq_cast(n, gdtype):
    """n % 4 == 0 takes the 16-byte-access kernel, the odd size the scalar one."""

    from research_b200.ops import native

    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda").to(gdtype)
    m, v = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    shadow = torch.empty(n, dtype=torch.bfloat16, device="cuda")
    pr = p.clone().requires_grad_(True)
    opt = torch.optim.AdamW([pr], lr=1e-2, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.1)
    for step in range(1, 4):
        pr.grad = g.float()
        opt.step()
        native.adamw(p, m, v, g, shadow, None, 1e-2, 0.9, 0.999, 1e-8, 0.1, step)
    assert torch.allclose(p, pr.detach(), atol=1e-5, rtol=1e-4)
    assert torch.allclose(shadow.float(), p, atol=1e-2, rtol=1e-2)
    out = torch.zeros(1, device="cuda")
    native.sumsq(g, out)
    assert math.isclose(out.item(), g.float().pow(2).sum().item(), rel_tol=1e-4)
    y = torch.empty(n, dtype=torch.bfloat16, device="cuda")
    native.cast_f32_bf16(p, y, 0.5)
    assert torch.allclose(y.float(), p * 0.5, atol=1e-2, rtol=1e-2)


@pytest.mark.parametrize("family", ["decoder", "trinity_moe", "trinity_moe_dion"])
def test_fast_muon_section_matches_reference_path(family):
    """The batched tcgen05 Muon step against the per-matrix PyTorch restatement of the same update
    (2-D matrices, row slices of fused parameters, and rank-3 expert stacks)."""

    import numpy as np

    from research_b200.config import run_spec_from_mapping
    from research_b200.contracts import Batch
    from research_b200.ops import native
    from research_b200.runtime.trainer import Trainer

    raw = {
        "run": {"id": "muon-parity"},
        "model": {"name": "decoder", "variant": "t", "vocab_size": 1024, "hidden_size": 256, "intermediate_size": 512,
                  "num_layers": 2, "num_heads": 2, "n_kv_heads": 1, "max_seq_len": 256, "init": "normal_0.02"},
        "optimizer": {"name": "muon", "weight_decay": 0.1, "grad_clip_norm": 1.0, "schedule": {"peak_lr": 1e-3}},
        "data": {"train_manifest": "unused.json"},
        "training": {"seq_len": 256, "global_batch_size": 2, "target_tokens": 2 * 256 * 4, "precision": "bf16"},
    }
    if family == "trinity_moe_dion":
        raw["optimizer"]["name"] = "dion"
    if family.startswith("trinity_moe"):
        raw["model"].update(name="trinity", num_layers=2, trinity={
            "initial_dense_layers": 1, "local_window": 128, "local_layers_per_global": 1, "norm_policy": "afmoe_dual",
            "moe": {"num_experts": 4, "top_k": 2, "expert_intermediate_size": 256, "num_shared_experts": 1}})
    rng = np.random.default_rng(0)
    ids = rng.integers(0, 1024, size=(2, 257)).astype(np.int32)
    batch = Batch(input_ids=ids[:, :-1], target_ids=ids[:, 1:], loss_mask=np.ones((2, 256), dtype=bool))
    results = []
    for fast in (True, False):
        trainer = Trainer(run_spec_from_mapping(raw), build_data=False)
        if not fast:
            trainer.optimizer._fast_muon_ok = lambda: False
        for _ in range(2):
            trainer.train_on([batch])
        native.check_status()
        results.append({e.name: trainer.store.master_view(trainer.store.section_of(e), e).clone()
                        for e in trainer.store.entries})
    lr = 1e-3
    for name, fast_w in results[0].items():
        slow_w = results[1][name]
        diff = (fast_w - slow_w).abs().max().item()
        if fast_w.dim() < 2 or any(k in name for k in ("embed", "lm_head", "norm")):
            # AdamW parameters: a near-zero gradient may flip sign between the two runs (their weights differ
            # after the first step), and Adam turns that into a full +-lr step each time
            assert diff <= 2 * 2 * lr + 1e-6, name
            continue
        # reference envelope for bf16 Newton-Schulz reorderings: update error <= 6e-4 at lr 1e-3 per step
        assert diff <= 2 * 6e-4 * (lr / 1e-3) + 1e-6, name


def test_qknorm_scales_that_the_predecessor_writes():
    """Scales straight out of a launch that lets its successor start early: bit for bit what they give with the device
    idle in between."""

    from research_b200.ops import native

    x, raw = _bf((200, 8 * 128), 51), [_bf((2, 128), 52 + i, 1.0 + i) for i in range(4)]
    ones, pos = torch.ones(128, device="cuda"), torch.arange(200, device="cuda", dtype=torch.int32)
    runs = []
    for idle in (True, False):
        got = []
        for i in range(32):
            scales = native.rmsnorm_fwd(raw[i % 4], ones, 1e-6)[0]
            if idle:
                torch.cuda.synchronize()
            out = torch.empty(200, 6 * 128, dtype=torch.bfloat16, device="cuda")
            native.qknorm_rope_fwd_qk(x, out, scales[0], scales[1], pos, 4, 2, 128, 1e-6, 10000.0, True)
            got.append(out)
        runs.append(got)
    native.check_status()
    assert all(torch.equal(u, v) for u, v in zip(*runs))
