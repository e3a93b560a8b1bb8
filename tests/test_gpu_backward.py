"""Backward pass of the windowed attention (the training form): the tcgen05 backward kernels against
``torch.autograd`` over the fp32 oracle, on the (T, window, documents, block window) grid of the forward tests;
bitwise run-to-run determinism; the norm / RoPE backward; the module under autograd against the reference-generated
fixture."""
import os

import numpy as np
import pytest
import torch

from gpu_util import assert_close_bf16, bf16_randn
from oracle import swa

pytestmark = pytest.mark.gpu
D = 128


def _prepared(B, T, H, seed):
    """RMS-normalised, rotated q, k and normalised v as bf16 (what the forward kernel consumes)."""
    q, k, v = (bf16_randn(B, T, H, D, seed=seed + i, device="cpu").float() for i in range(3))
    cos, sin = swa.rope_tables(D, T)
    qn, kn, vn = swa.qkv_transform(q, k, v, cos, sin, swa.FP32_EPS)
    return qn.bfloat16(), kn.bfloat16(), vn.bfloat16()


def _check_grads(got, ref, what, cancelling=False):
    """bf16 bar of the forward tests, plus relative L2 <= 2e-2.  ``cancelling``: windows of one or two keys, where the
    exact dq and dk are (nearly) zero as the difference dP - delta of two terms of magnitude |dO||v| ~ 10..40: delta
    is formed from the bf16 output O, which carries the forward's bf16 rounding of P (2^-9 relative), so an
    absolute error of 2^-8 * max|dP| * scale * max|k| ~ 0.05 remains -- the same in any implementation that takes
    delta from the stored output."""
    for g, r, n in zip(got, ref, ("dq", "dk", "dv")):
        if cancelling and n != "dv":
            assert_close_bf16(g, r, f"{what} {n}", max_tol=0.1, mean_tol=0.01)
            continue
        assert_close_bf16(g, r, f"{what} {n}")
        rel = ((g.float().cpu() - r).norm() / r.norm().clamp_min(1e-20)).item()
        assert rel <= 2e-2, f"{what} {n}: relative L2 {rel}"


@pytest.mark.parametrize("T,window", [(128, None), (300, 64), (256, 128), (257, 1), (640, 200), (1000, 129), (131, 500), (512, 2)])
def test_attend_backward_matches_autograd_oracle(T, window):
    from daisy_b200 import ops
    B, H = 2, 2
    q, k, v = _prepared(B, T, H, seed=T)
    d_o = bf16_randn(B, T, H, D, seed=T + 9, device="cpu")
    y_ref, *ref = swa.attend_backward(q.float(), k.float(), v.float(), d_o.float(), window)
    qc, kc, vc, gc = (t.cuda() for t in (q, k, v, d_o))
    y, lse = ops.swa_attend(qc, kc, vc, window, bounded_qk=True, return_lse=True)
    got = ops.swa_attend_bwd(qc, kc, vc, y, gc, lse, window)
    ops.check_device_status("cuda")
    assert_close_bf16(y, y_ref, "forward with lse")
    _check_grads(got, ref, f"T={T} W={window}", cancelling=window is not None and window <= 2)
    # the general (running-maximum) forward form stores the same quantity
    y2, lse2 = ops.swa_attend(qc, kc, vc, window, bounded_qk=False, return_lse=True)
    assert (lse2 - lse).abs().max().item() <= 2e-2
    again = ops.swa_attend_bwd(qc, kc, vc, y, gc, lse, window)
    assert all(torch.equal(a, b) for a, b in zip(got, again)), "backward is not run-to-run deterministic"


@pytest.mark.parametrize("T,window,n_docs,per_batch", [(384, 100, 3, False), (700, None, 12, False), (512, 64, 5, True)])
def test_attend_backward_with_documents(T, window, n_docs, per_batch):
    from daisy_b200 import ops
    B, H = 2, 2
    q, k, v = _prepared(B, T, H, seed=T + 1)
    d_o = bf16_randn(B, T, H, D, seed=T + 5, device="cpu")
    g = torch.Generator().manual_seed(T)
    rows = []
    for _ in range(B if per_batch else 1):
        cuts = torch.sort(torch.randperm(T - 1, generator=g)[:n_docs - 1] + 1).values
        ds = torch.zeros(T, dtype=torch.int32)
        for c in cuts.tolist():
            ds[c:] = c
        rows.append(ds)
    ds = torch.stack(rows) if per_batch else rows[0]
    _, *ref = swa.attend_backward(q.float(), k.float(), v.float(), d_o.float(), window, doc_start=ds)
    qc, kc, vc, gc = (t.cuda() for t in (q, k, v, d_o))
    y, lse = ops.swa_attend(qc, kc, vc, window, bounded_qk=True, doc_start=ds.cuda(), return_lse=True)
    got = ops.swa_attend_bwd(qc, kc, vc, y, gc, lse, window, doc_start=ds.cuda())
    ops.check_device_status("cuda")
    _check_grads(got, ref, f"docs T={T}")


@pytest.mark.parametrize("T,wb,n_docs", [(512, 2, 1), (768, 1, 4), (640, 3, 6)])
def test_attend_backward_block_window_training_form(T, wb, n_docs):
    """The flex-attention form: the window counts 128-token key blocks (models/daisy/daisy_core.py:182-229)."""
    from daisy_b200 import ops
    B, H = 1, 2
    q, k, v = _prepared(B, T, H, seed=T + 2)
    d_o = bf16_randn(B, T, H, D, seed=T + 6, device="cpu")
    g = torch.Generator().manual_seed(T + wb)
    ds = torch.zeros(T, dtype=torch.int32)
    for c in torch.sort(torch.randperm(T - 1, generator=g)[:n_docs - 1] + 1).values.tolist():
        ds[c:] = c
    _, *ref = swa.attend_backward(q.float(), k.float(), v.float(), d_o.float(), None, doc_start=ds, window_blocks=wb)
    qc, kc, vc, gc = (t.cuda() for t in (q, k, v, d_o))
    y, lse = ops.swa_attend(qc, kc, vc, wb, bounded_qk=True, doc_start=ds.cuda(), window_in_blocks=True, return_lse=True)
    got = ops.swa_attend_bwd(qc, kc, vc, y, gc, lse, wb, doc_start=ds.cuda(), window_in_blocks=True)
    ops.check_device_status("cuda")
    _check_grads(got, ref, f"block window T={T} wb={wb}")


@pytest.mark.parametrize("T,window,in_blocks,docs", [(128, None, False, False), (129, 1, False, False), (300, 130, False, True),
                                                     (700, 127, False, False), (640, 2, True, True), (1000, None, False, True)])
def test_attend_backward_workspaces(T, window, in_blocks, docs):
    """dZ kept for dQ (workspace for all (batch, head) pairs, for two of six, i.e. several rounds, for one) or formed again
    (delta alone): the same dK, dV and, of the first three, dQ bit for bit; both dQ at the bf16 bar of the oracle."""
    from daisy_b200 import _lib, ops
    B, H = 2, 3
    q, k, v = _prepared(B, T, H, seed=T + 3)
    d_o = bf16_randn(B, T, H, D, seed=T + 7, device="cpu")
    ds = torch.zeros(T, dtype=torch.int32)
    if docs:
        for c in (T // 5, T // 3, T - 60):
            ds[c:] = c
    _, *ref = swa.attend_backward(q.float(), k.float(), v.float(), d_o.float(), None if in_blocks else window,
                                  doc_start=ds if docs else None, window_blocks=window if in_blocks else None)
    q, k, v, d_o = (t.cuda() for t in (q, k, v, d_o))
    doc = ds.cuda() if docs else None
    y, lse = ops.swa_attend(q, k, v, window, bounded_qk=True, doc_start=doc, window_in_blocks=in_blocks, return_lse=True)
    L, flags = _lib.lib(), _lib.WINDOW_BLOCKS if in_blocks else 0
    full = L.daisy_b200_swa_attend_bwd_workspace_bytes_full(B, T, H, window or 0, flags)
    delta = -(-L.daisy_b200_swa_attend_bwd_workspace_bytes(B, T, H) // 1024) * 1024
    one = (full - delta) // (B * H)
    assert one % 32768 == 0 and one > 0
    st = (T * H * D, H * D, D) * 5
    got = []
    for size in (full, delta + 2 * one, delta + one, delta):
        out = [torch.full((B, T, H, D), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3)]
        ws = torch.full((size + 4096,), 0xff, dtype=torch.uint8, device="cuda")          # NaN images; guard behind the workspace
        rc = L.daisy_b200_swa_attend_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), y.data_ptr(), d_o.data_ptr(), *st, lse.data_ptr(),
                                         *(t.data_ptr() for t in out), B, T, H, D, window or 0, 0.12, doc.data_ptr() if docs else None, 0,
                                         flags, ws.data_ptr(), size, ops.status_word(q.device).data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        ops.check_device_status("cuda")
        assert bool((ws[size:] == 0xff).all())
        got.append(out)
    for out in got[1:]:
        assert torch.equal(out[1], got[0][1]) and torch.equal(out[2], got[0][2])
    assert torch.equal(got[1][0], got[0][0]) and torch.equal(got[2][0], got[0][0])
    for out in (got[0], got[3]):
        _check_grads(out, ref, f"T={T} W={window}", cancelling=not in_blocks and window == 1)


def test_prep_backward_matches_autograd():
    """Norm / RoPE backward on strided views of a merged projection."""
    from daisy_b200 import ops
    B, T, H = 2, 150, 3
    qkv = bf16_randn(B, T, 3 * H, D, seed=1)
    q, k, v = qkv.chunk(3, dim=-2)
    gs = [bf16_randn(B, T, H, D, seed=20 + i) for i in range(3)]
    cos, sin = swa.rope_tables(D, T)
    leaves = [t.float().cpu().requires_grad_(True) for t in (q, k, v)]
    outs = swa.qkv_transform(*leaves, cos, sin, swa.FP32_EPS)
    sum((o * g.float().cpu()).sum() for o, g in zip(outs, gs)).backward()
    got = ops.qkv_prep_bwd(q, k, v, cos.cuda(), sin.cuda(), *gs, swa.FP32_EPS)
    for g_, leaf, n in zip(got, leaves, "qkv"):
        assert_close_bf16(g_, leaf.grad, f"d{n} raw")


def test_module_forward_under_autograd_matches_reference_fixture(golden_dir):
    """``loss.backward()`` through ``B200CausalSelfAttention.forward`` with the document mask: input and weight
    gradients against the reference module's own autograd results (fp32, CPU)."""
    from daisy_b200 import B200CausalSelfAttention, WindowMask
    d = np.load(os.path.join(golden_dir, "csa_backward_small.npz"))
    attn = B200CausalSelfAttention(dim=256, num_heads=2, head_dim=128, max_seq_len=256).cuda()
    attn.norm_eps = swa.FP32_EPS
    with torch.no_grad():
        attn.qkvo_w.copy_(torch.from_numpy(d["qkvo_w"]).to(attn.qkvo_w.dtype))
    x = torch.from_numpy(d["x"]).cuda().bfloat16().requires_grad_(True)
    mask = WindowMask.from_tokens(torch.from_numpy(d["seq"]).cuda(), int(d["window"]), int(d["eos"]))
    y = attn(x, None, attn_mask=mask)
    assert y.requires_grad
    (y.float() * torch.from_numpy(d["cot"]).cuda()).sum().backward()
    assert_close_bf16(y.detach(), torch.from_numpy(d["y"]), "y", max_tol=4e-2, mean_tol=4e-3)
    assert_close_bf16(x.grad, torch.from_numpy(d["dx"]), "dx", max_tol=4e-2, mean_tol=4e-3)
    assert_close_bf16(attn.qkvo_w.grad, torch.from_numpy(d["dw"]), "dw", max_tol=4e-2, mean_tol=4e-3)
    # and the inference route computes the same forward
    with torch.inference_mode():
        y_inf = attn(x.detach(), None, attn_mask=mask)
    assert_close_bf16(y_inf, y.detach().float().cpu(), "inference vs training forward", max_tol=3e-2, mean_tol=3e-3)


def test_value_embedding_layer_under_autograd():
    """A layer that receives a value embedding, trained: the gate ``v = s(g_ve) norm(v) + (1 - s(g_ve)) ve``
    (models/daisy/attention.py:132-135) sits between the norm and the attention, and ``loss.backward()`` must reach x, the
    merged weights, the gate parameter and ve.  Compared with ``torch.autograd`` over the fp32 oracle functions."""
    from daisy_b200 import B200CausalSelfAttention, WindowMask
    os.environ["DISABLE_O_ZERO_INIT"] = "1"
    torch.manual_seed(3)
    H, T, W = 2, 200, 64
    m = B200CausalSelfAttention(H * D, H, D, receives_ve=True, layer_idx=2).cuda()
    m.norm_eps = swa.FP32_EPS
    x = torch.randn(1, T, H * D, device="cuda").bfloat16().requires_grad_(True)
    ve = torch.randn(1, T, H * D, device="cuda").bfloat16().requires_grad_(True)
    cot = torch.randn(1, T, H * D, device="cuda")
    y = m(x, ve, attn_mask=WindowMask(W))
    assert y.requires_grad
    (y.float() * cot).sum().backward()
    # oracle: the same computation in fp32 on the CPU
    xo = x.detach().float().cpu().requires_grad_(True)
    vo = ve.detach().float().cpu().requires_grad_(True)
    wo = m.qkvo_w.detach().float().cpu().requires_grad_(True)
    go = m.g_ve.detach().float().cpu().requires_grad_(True)
    q, k, v = swa.project_qkv(xo, wo, H, D)
    cos, sin = swa.rope_tables(D, T)
    qn, kn, vn = swa.qkv_transform(q, k, v, cos, sin, swa.FP32_EPS)
    gate = torch.sigmoid(go)
    vn = gate * vn + (1 - gate) * vo.view_as(vn)
    yo = swa.attend_windowed(qn, kn, vn, W).reshape(1, T, H * D) @ wo[3].t()
    (yo * cot.cpu()).sum().backward()
    assert_close_bf16(y.detach(), yo.detach(), "y", max_tol=4e-2, mean_tol=4e-3)
    assert_close_bf16(x.grad, xo.grad, "dx", max_tol=4e-2, mean_tol=4e-3)
    assert_close_bf16(ve.grad, vo.grad, "d ve", max_tol=4e-2, mean_tol=4e-3)
    assert_close_bf16(m.qkvo_w.grad, wo.grad, "dw", max_tol=4e-2, mean_tol=4e-3)
    g_got, g_ref = m.g_ve.grad.float().cpu().reshape(-1), go.grad.reshape(-1)
    assert torch.allclose(g_got, g_ref, rtol=5e-2, atol=5e-2 * float(g_ref.abs().max()) + 1e-3), (g_got, g_ref)
    # the inference route computes the same forward
    with torch.inference_mode():
        y_inf = m(x.detach(), ve.detach(), attn_mask=WindowMask(W))
    assert_close_bf16(y_inf, y.detach().float().cpu(), "inference vs training forward", max_tol=3e-2, mean_tol=3e-3)


@pytest.mark.parametrize("B,T,H", [(1, 40, 1), (2, 33, 1), (1, 63, 3), (3, 129, 6)])
def test_gated_layer_backward_ragged_rows(B, T, H):
    """The row-wise gradient pass takes 64 (token, head) rows a block, two to a thread group: fewer rows than a block, remainders
    of either kind, against ``torch.autograd`` over the fp32 oracle."""
    from daisy_b200 import B200CausalSelfAttention, WindowMask
    os.environ["DISABLE_O_ZERO_INIT"] = "1"
    torch.manual_seed(T)
    m = B200CausalSelfAttention(H * D, H, D, receives_ve=True, layer_idx=2).cuda()
    m.norm_eps = swa.FP32_EPS
    x = torch.randn(B, T, H * D, device="cuda").bfloat16().requires_grad_(True)
    ve = torch.randn(B, T, H * D, device="cuda").bfloat16().requires_grad_(True)
    cot = torch.randn(B, T, H * D, device="cuda")
    (m(x, ve, attn_mask=WindowMask(50)).float() * cot).sum().backward()
    xo, vo, wo = (t.detach().float().cpu().requires_grad_(True) for t in (x, ve, m.qkvo_w))
    q, k, v = swa.project_qkv(xo, wo, H, D)
    cos, sin = swa.rope_tables(D, T)
    qn, kn, vn = swa.qkv_transform(q, k, v, cos, sin, swa.FP32_EPS)
    gate = torch.sigmoid(m.g_ve.detach().float().cpu())
    vn = gate * vn + (1 - gate) * vo.view_as(vn)
    yo = swa.attend_windowed(qn, kn, vn, 50).reshape(B, T, H * D) @ wo[3].t()
    (yo * cot.cpu()).sum().backward()
    for got, ref, n in ((x.grad, xo.grad, "dx"), (ve.grad, vo.grad, "d ve"), (m.qkvo_w.grad, wo.grad, "dw")):
        assert_close_bf16(got, ref, n, max_tol=4e-2, mean_tol=4e-3)


@pytest.mark.parametrize("changed", ["x", "ve", "g_ve", "qkvo_w", "doc_start", None])
def test_in_place_change_before_backward_raises(changed):
    """What the backward reads again is saved as it was handed in: an in-place change between forward and backward is
    refused, and without one the gradients do not depend on saved-tensor hooks that move what was saved."""
    from daisy_b200 import B200CausalSelfAttention, WindowMask
    os.environ["DISABLE_O_ZERO_INIT"] = "1"
    torch.manual_seed(1)
    H, T = 2, 96
    m = B200CausalSelfAttention(H * D, H, D, receives_ve=True, layer_idx=2).cuda()
    leaf = torch.randn(1, T, H * D, device="cuda").bfloat16().requires_grad_(True)
    ve = torch.randn(1, T, H * D, device="cuda").bfloat16()
    doc = torch.zeros(T, dtype=torch.int32, device="cuda")

    def forward():
        x = leaf * 1                                                       # not a leaf: it may be changed in place
        return x, m(x, ve, attn_mask=WindowMask(40, doc))

    if changed is None:
        wrt = [leaf, m.qkvo_w, m.g_ve]
        _, y = forward()
        ref = torch.autograd.grad(y.sum(), wrt)
        with torch.autograd.graph.save_on_cpu():
            _, y = forward()
        assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y.sum(), wrt), ref))
        with torch.inference_mode():
            ve = ve.clone()                                                # an embedding made in inference mode
        _, y = forward()
        assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y.sum(), wrt), ref))
        return
    x, y = forward()
    with torch.no_grad():
        dict(x=x, ve=ve, g_ve=m.g_ve, qkvo_w=m.qkvo_w, doc_start=doc)[changed].add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()


def test_training_layer_takes_any_alignment():
    """x, ve and the weights at addresses and strides that no 16-byte load can fetch against the call on aligned copies: the
    same y; gradients from the library's products, whose fp32 sums may go in another order there, up to one bf16 rounding
    (2^-8 of a value)."""
    from daisy_b200 import B200CausalSelfAttention, WindowMask
    os.environ["DISABLE_O_ZERO_INIT"] = "1"
    torch.manual_seed(2)
    H, T = 2, 96
    dim = H * D
    m = B200CausalSelfAttention(dim, H, D, receives_ve=True, layer_idx=2).cuda()
    w, x, ve = m.qkvo_w.detach().clone(), *(torch.randn(2, T, dim, device="cuda").bfloat16() for _ in range(2))

    def off(t):                                                            # the same values one element further on
        return torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t)

    wide = torch.empty(2, T, dim + 3, dtype=x.dtype, device="cuda")[..., :dim].copy_(x)      # rows 2 * 259 bytes apart
    ref = None
    for x_, ve_, w_ in ((x, ve, w), (off(x), ve, w), (wide, ve, w), (x, off(ve), w), (x, ve, off(w))):
        x_, ve_ = x_.requires_grad_(True), ve_.requires_grad_(True)
        m.qkvo_w = torch.nn.Parameter(w_)
        y = m(x_, ve_, attn_mask=WindowMask(40))
        got = [y.detach(), *torch.autograd.grad(y.float().square().sum(), [x_, ve_, m.qkvo_w, m.g_ve])]
        ref = ref or got
        assert torch.equal(got[0], ref[0])
        assert all(((a.float() - b.float()).norm() / b.float().norm()).item() <= 2 ** -8 for a, b in zip(got[1:], ref[1:]))


def test_backward_without_room_for_the_images():
    """Where the allocator has no room for the dZ images (268 MB here) the layer's and the operator's backward take the workspace
    without them: the same dK and dV bits, dQ from the scores formed again, one rounding of dZ to bf16 either way (2^-8)."""
    from daisy_b200 import B200CausalSelfAttention, WindowMask, ops
    os.environ["DISABLE_O_ZERO_INIT"] = "1"
    torch.manual_seed(4)
    H, T = 2, 8192
    m = B200CausalSelfAttention(H * D, H, D, receives_ve=False, layer_idx=None, max_seq_len=T).cuda()
    x = torch.randn(1, T, H * D, device="cuda").bfloat16().requires_grad_(True)
    q, k, v, d_o = (torch.randn(1, T, H, D, device="cuda").bfloat16() for _ in range(4))
    q, k = (t / t.float().square().mean(-1, keepdim=True).sqrt().to(t.dtype) for t in (q, k))
    o, lse2 = ops.swa_attend(q, k, v, T, 0.12, return_lse=True)

    def both():
        y = m(x, None, attn_mask=WindowMask(T))
        return [*torch.autograd.grad(y, [x, m.qkvo_w], torch.ones_like(y)), *ops.swa_attend_bwd(q, k, v, o, d_o, lse2, T, 0.12)]
    ref = both()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (200 << 20)) / total)
        with pytest.raises(torch.cuda.OutOfMemoryError):
            torch.empty(268 << 20, dtype=torch.uint8, device="cuda")
        got = both()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    ops.check_device_status("cuda")
    assert torch.equal(got[3], ref[3]) and torch.equal(got[4], ref[4])
    assert all(((a.float() - b.float()).norm() / b.float().norm()).item() <= 2 ** -8 for a, b in zip(got, ref))


def test_backward_asks_once_for_room_that_is_refused():
    """A refused workspace costs the allocator its cached blocks and waits for the device: the operator and the layer, whose images
    are of one size, ask for it once between them and not in every call, and go on asking for what is smaller."""
    from daisy_b200 import B200CausalSelfAttention, WindowMask, ops
    os.environ["DISABLE_O_ZERO_INIT"] = "1"
    torch.manual_seed(5)
    H, T = 2, 16384
    m = B200CausalSelfAttention(H * D, H, D, receives_ve=False, layer_idx=None, max_seq_len=T).cuda()
    x = torch.randn(1, T, H * D, device="cuda").bfloat16().requires_grad_(True)

    def call(t):
        q, k, v, o, d_o = (torch.zeros(1, t, H, D, device="cuda", dtype=torch.bfloat16) for _ in range(5))
        return ops.swa_attend_bwd(q, k, v, o, d_o, torch.zeros(1, H, t, device="cuda"), None)

    def layer():
        y = m(x, None, attn_mask=WindowMask(T))
        torch.autograd.grad(y, [x, m.qkvo_w], torch.ones_like(y))
    layer()
    call(1024)
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    refused = lambda: torch.cuda.memory_stats()["num_alloc_retries"]
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (400 << 20)) / total)
        before = refused()
        for _ in range(4):
            call(T)
            layer()
        assert refused() - before <= 1                           # none where a test before this one met the refusal
        torch.cuda.reset_peak_memory_stats()
        held = torch.cuda.memory_allocated()
        call(1024)
        assert torch.cuda.max_memory_allocated() - held > 6 << 20     # inputs and gradients are 4 MB; images 2 x 36 of 32 KB at least
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    ops.check_device_status("cuda")
