"""The single-launch decode step (csrc/swa_token.cu) against the CPU oracle, at the edges of its partition: one and many
layers, batch 1 to 16, one row tile or several, contexts of 0, 1, 15 .. 17 and many rows, a wrapped ring, fp16 rings."""
import pytest
import torch

from gpu_util import assert_close_bf16
from oracle import swa

pytestmark = pytest.mark.gpu
D = 128


def _setup(B, H, L, cap, f16, seed=0):
    g = torch.Generator().manual_seed(seed)
    dim = H * D
    w = [(torch.randn(4, dim, dim, generator=g) * dim ** -0.5).bfloat16() for _ in range(L)]
    ring = [torch.randn(L, B, H, cap, D, generator=g).to(torch.float16 if f16 else torch.bfloat16) for _ in range(2)]
    return w, ring, torch.randn(B, 1, dim, generator=g).bfloat16()


def _oracle(w, rk, rv, x, t, cap, window, cos, sin, eps):
    B, _, dim = x.shape
    H = dim // D
    qkv = (x.float() @ w[:3].flatten(end_dim=1).float().T).bfloat16().float().view(B, 1, 3 * H, D)
    idx = torch.arange(t - min(t, cap), t) % cap
    y, k, v = swa.decode_step(*qkv.chunk(3, dim=-2), rk[:, :, idx].transpose(1, 2).float(), rv[:, :, idx].transpose(1, 2).float(), t, window,
                              cos, sin, eps=eps)
    return (y.reshape(B, 1, dim).bfloat16().float() @ w[3].float().T).bfloat16(), k, v


@pytest.mark.parametrize("B,H,L,t,cap,window,f16", [
    (1, 1, 1, 0, 48, 16, False), (1, 3, 2, 1, 48, 16, False), (2, 2, 1, 16, 48, 17, True), (3, 5, 2, 100, 48, 100, False),
    (1, 16, 2, 3000, 2048, 2048, False), (8, 6, 1, 700, 512, 300, True), (9, 4, 2, 77, 64, 18, False), (16, 16, 1, 130, 64, 64, False),
    (1, 2, 17, 40, 32, 24, False),
])
def test_token_step_matches_oracle(B, H, L, t, cap, window, f16):
    from daisy_b200 import ops
    from daisy_b200._lib import QKV_DEFAULT, WRITE_RING
    from daisy_b200._native import ext
    w, (rk, rv), x = _setup(B, H, L, cap, f16)
    eps = float(torch.finfo(torch.bfloat16).eps)
    cos, sin = swa.rope_tables(D, t + 2)
    dev = [a.cuda() for a in w], rk.cuda(), rv.cuda(), x.cuda(), cos.cuda(), sin.cuda()
    assert ext().token_step_supported(B, H, L)
    t_dev, adv = torch.tensor([t], device="cuda"), torch.tensor([t], device="cuda")
    args = lambda k, v, pos, d, a: (dev[3], dev[0], [dev[4]] * L, [dev[5]] * L, k, v, pos, d, a, window, 0.12, eps, QKV_DEFAULT | WRITE_RING,
                                    None, None, None, None, None, None)
    k1, v1 = dev[1].clone(), dev[2].clone()
    y = ext().token_step(*args(k1, v1, t, None, adv))
    k2, v2 = dev[1].clone(), dev[2].clone()
    y2 = ext().token_step(*args(k2, v2, 0, t_dev, None))
    ops.check_device_status("cuda")
    assert torch.equal(y, y2) and torch.equal(k1, k2) and torch.equal(v1, v2), "position on the device"
    assert int(adv) == t + 1 and int(t_dev) == t
    h = x
    for l in range(L):
        h, k, v = _oracle(w[l], rk[l], rv[l], h, t, cap, window, cos, sin, eps)
        if l == 0:
            got_k, got_v = k1[0, :, :, t % cap].float().cpu(), v1[0, :, :, t % cap].float().cpu()
            assert_close_bf16(got_k, k[:, 0], "new k row")
            assert_close_bf16(got_v, v[:, 0], "new v row")
    rel = ((y.float().cpu() - h.float()).norm() / h.float().norm()).item()
    assert rel < 1e-2 * max(1.0, L ** 0.5), rel
    mask = torch.ones(cap, dtype=torch.bool)
    mask[t % cap] = False
    assert torch.equal(k1[:, :, :, mask].cpu(), rk[:, :, :, mask]) and torch.equal(v1[:, :, :, mask].cpu(), rv[:, :, :, mask])


@pytest.mark.parametrize("t,cap,window", [(5, 64, 40), (16, 64, 40), (47, 64, 48), (100, 64, 20), (130, 64, 50), (63, 64, 64), (0, 64, 40)])
@pytest.mark.parametrize("f16", [False, True])
def test_token_step_ignores_rows_outside_the_context(t, cap, window, f16):
    """Ring slots outside the context hold infinities and NaN (a ring that another sequence has used): the same bits as over
    zeros, with the context ending inside a piece of 16 rows, at one, at the ring's end, and wrapped."""
    from daisy_b200 import ops
    from daisy_b200._lib import QKV_DEFAULT
    from daisy_b200._native import ext
    B, H = 2, 3
    w, ring, x = _setup(B, H, 1, cap, f16, seed=t)
    cos, sin = (a.cuda() for a in swa.rope_tables(D, t + 1))
    keep = torch.zeros(cap, dtype=torch.bool)
    keep[torch.arange(t - min(t, cap, window - 1), t) % cap] = True
    ys = []
    for fill in ((0.0, 0.0), (float("nan"), float("inf")), (float("-inf"), float("nan"))):
        rk, rv = (r.clone() for r in ring)
        rk[:, :, :, ~keep], rv[:, :, :, ~keep] = fill
        ys.append(ext().token_step(x.cuda(), [w[0].cuda()], [cos], [sin], rk.cuda(), rv.cuda(), t, None, None, window, 0.12, 1e-6, QKV_DEFAULT,
                                   None, None, None, None, None, None))
    ops.check_device_status("cuda")
    assert torch.isfinite(ys[0].float()).all() and all(torch.equal(y, ys[0]) for y in ys[1:])


@pytest.mark.parametrize("B,H", [(1, 2), (3, 2), (1, 1)])
def test_token_step_of_narrow_layers_repeats(B, H):
    """Layers of which some CTAs own no output row (128 and 256 channels), sixteen of them: the same bits in a hundred launches."""
    from daisy_b200 import ops
    from daisy_b200._lib import QKV_DEFAULT
    from daisy_b200._native import ext
    L, cap, t = 16, 64, 500
    w, (rk, rv), x = _setup(B, H, L, cap, False, seed=7)
    cos, sin = (a.cuda() for a in swa.rope_tables(D, t + 1))
    w, rk, rv, x = [a.cuda() for a in w], rk.cuda(), rv.cuda(), x.cuda()
    ys = [ext().token_step(x, w, [cos] * L, [sin] * L, rk, rv, t, None, None, 48, 0.12, 1e-6, QKV_DEFAULT, None, None, None, None, None, None)
          for _ in range(100)]
    ops.check_device_status("cuda")
    assert all(torch.equal(y, ys[0]) for y in ys[1:])


@pytest.mark.parametrize("B,H,bias", [(1, 1, False), (3, 6, True), (8, 16, False), (9, 5, True), (17, 2, False)])
def test_kimi_token_step_continues_a_prefill(B, H, bias):
    """The single-launch Kimi step (csrc/kda_token.cu) after a prefill of T tokens against a prefill of T + 1: the output,
    the recurrent state and the convolution states; batches that are one, several and more than sixteen rows."""
    from daisy_b200 import B200KimiLinearSelfAttention, ops
    torch.manual_seed(B * 100 + H)
    layer = B200KimiLinearSelfAttention(H * D, H, 4096, D, conv_bias=bias).cuda()
    T = 70
    x = torch.randn(B, T + 1, H * D, device="cuda", dtype=torch.bfloat16)
    with torch.inference_mode():
        ref, _, _ = layer.prefill(x)
        rec, conv = layer._recurrent_state.clone(), [c.clone() for c in layer._conv_state]
        layer.reset_history()
        layer.prefill(x[:, :T])
        assert layer._token_step(x[:, T:], torch.empty(B, 1, H * D, device="cuda", dtype=torch.bfloat16)) is not None
        layer.reset_history()
        layer.prefill(x[:, :T])
        y, _, _ = layer.step(x[:, T:])
    ops.check_device_status("cuda")
    assert_close_bf16(y, ref[:, T:], "y", max_tol=3e-2, mean_tol=3e-3)
    assert ((layer._recurrent_state - rec).norm() / rec.norm()).item() < 5e-3
    for a, b in zip(layer._conv_state, conv):
        assert torch.equal(a[..., :3], b[..., :3]), "the carried inputs move up"
        assert_close_bf16(a, b, "the new input")


@pytest.mark.parametrize("B,H,bias", [(17, 1, True), (33, 3, False), (64, 16, True)])
def test_kimi_batch_step_matches_row_launches(B, H, bias):
    """Above 16 rows (kda_batch_kernel between GEMMs) against the single launch on as many rows at a time as it takes (16, and 168
    (row, head) pairs): the convolution states bit for bit but for the new input, everything else to the order of fp32 sums under
    bf16 roundings."""
    from daisy_b200 import B200KimiLinearSelfAttention, ops
    torch.manual_seed(B)
    layer = B200KimiLinearSelfAttention(H * D, H, 4096, D, conv_bias=bias).cuda()
    x = torch.randn(B, 30, H * D, device="cuda", dtype=torch.bfloat16)
    with torch.inference_mode():
        layer.prefill(x[:, :29])
        rec, conv = layer._recurrent_state.clone(), [c.clone() for c in layer._conv_state]
        y, _, _ = layer.step(x[:, 29:])
        got = (y, layer._recurrent_state, *layer._conv_state)
        ys = []
        n = min(16, 168 // H)
        for b in range(0, B, n):
            layer._recurrent_state, layer._conv_state = rec[b:b + n].clone(), tuple(c[b:b + n].clone() for c in conv)
            ys.append((layer.step(x[b:b + n, 29:])[0], layer._recurrent_state, *layer._conv_state))
    ops.check_device_status("cuda")
    ref = [torch.cat(t) for t in zip(*ys)]
    assert_close_bf16(got[0], ref[0], "y", max_tol=3e-2, mean_tol=3e-3)
    assert ((got[1] - ref[1]).norm() / ref[1].norm()).item() < 5e-3
    for a, b in zip(got[2:], ref[2:]):
        assert torch.equal(a[..., :3], b[..., :3])
        assert_close_bf16(a, b, "the new input")


@pytest.mark.parametrize("B,H", [(11, 16), (16, 16), (15, 12), (10, 16), (14, 12)])
def test_kimi_step_either_side_of_the_line_between_its_routes(B, H):
    """The most (batch, head) pairs of the single launch and the fewest of the four, in turn with single launches of one row: they
    share a workspace, whose words the four launches' scratch must leave alone."""
    from daisy_b200 import B200KimiLinearSelfAttention, ops
    torch.manual_seed(B)
    layer = B200KimiLinearSelfAttention(H * D, H, 4096, D).cuda()
    x = torch.randn(B, 30, H * D, device="cuda", dtype=torch.bfloat16)
    with torch.inference_mode():
        layer.prefill(x[:, :29])
        rec, conv = layer._recurrent_state.clone(), [c.clone() for c in layer._conv_state]

        def step(b, n):
            layer._recurrent_state, layer._conv_state = rec[b:b + n].clone(), tuple(c[b:b + n].clone() for c in conv)
            return (layer.step(x[b:b + n, 29:])[0], layer._recurrent_state, *layer._conv_state)
        got, ys = step(0, B), []
        for b in range(B):
            ys.append(step(b, 1))
            again = step(0, B)
            assert all(torch.equal(a, g) for a, g in zip(again, got))
    ops.check_device_status("cuda")
    ref = [torch.cat(t) for t in zip(*ys)]
    assert_close_bf16(got[0], ref[0], "y", max_tol=3e-2, mean_tol=3e-3)
    assert ((got[1] - ref[1]).norm() / ref[1].norm()).item() < 5e-3
    for a, b in zip(got[2:], ref[2:]):
        assert torch.equal(a[..., :3], b[..., :3])
        assert_close_bf16(a, b, "the new input")
