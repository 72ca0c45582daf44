"""The native front of the operators (csrc/torch_binding.cpp) and the kernel paths it opened: dilated
1-D layouts folded into tensor-map axes, narrow head dims in the backward, layers as one autograd
node, column sums. Against the oracle with the 16-bit tolerance of the other files (2e-2 of the
largest entry), or against the Python front."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import natten_b200 as nb
import natten_b200._lib as L
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,ks,st,di,ca,hq,hkv,D,n_extra,B", [
    ((1200,), (33,), (1,), (3,), (True,), 2, 2, 64, 0, 2),      # length a multiple of the dilation
    ((1201,), (65,), (4,), (3,), (False,), 2, 1, 128, 20, 2),   # two kinds of groups, extra tokens
    ((515,), (2,), (1,), (257,), (False,), 1, 1, 32, 0, 1),     # one or two keys per group, folded + narrow
    ((777,), (40,), (1,), (16,), (True,), 4, 2, 24, 130, 2),    # narrow, ragged, GQA, extras
    ((300,), (33,), (1,), (2,), (False,), 2, 2, 64, 0, 2),      # folded at dilation 2 ...
    ((301,), (33,), (1,), (2,), (False,), 2, 2, 64, 0, 2),      # ... and the strided box beside it
    ((33, 30), (3, 5), (1, 2), (3, 2), (False, True), 4, 2, 8, 0, 2),
    ((31, 29), (7, 7), (1, 1), (1, 1), (False, False), 3, 3, 40, 33, 3),
    ((5, 12, 20), (3, 5, 6), (1, 1, 2), (1, 1, 1), (True, False, False), 2, 2, 80, 0, 1),
    ((5, 12, 20), (3, 5, 6), (1, 1, 2), (1, 1, 1), (True, False, False), 2, 2, 120, 9, 1),
])
def test_folded_and_narrow_problems(shape, ks, st, di, ca, hq, hkv, D, n_extra, B):
    torch.manual_seed(41)
    fn = {1: nb.na1d, 2: nb.na2d, 3: nb.na3d}[len(shape)]
    q, d_out = (torch.randn(B, *shape, hq, D).half() for _ in range(2))
    k, v = (torch.randn(B, *shape, hkv, D).half() for _ in range(2))
    extras = [torch.randn(B, n_extra, hkv, D).half() for _ in range(2)] if n_extra else []
    leaves = [t.cuda().requires_grad_() for t in [q, k, v] + extras]
    add = dict(additional_keys=leaves[3], additional_values=leaves[4]) if n_extra else {}
    before = L.launches
    out, lse = fn(*leaves[:3], ks, st, di, ca, return_lse=True, **add)
    assert "NaFunction" in out.grad_fn.name()
    out.backward(d_out.cuda())
    assert L.launches - before >= 4 and L.device_status() == 0
    f = [t.float().numpy() for t in (q, k, v)]
    ex = dict(add_k=extras[0].float().numpy(), add_v=extras[1].float().numpy()) if n_extra else {}
    want_o, want_l = oracle.na_forward(*f, ks, st, di, ca, **ex)
    assert np.abs(out.detach().float().cpu().numpy() - want_o).max() <= 2e-2
    assert np.abs(lse.detach().cpu().numpy() - want_l).max() <= 2e-2
    want = oracle.na_backward(*f, d_out.float().numpy(), ks, st, di, ca, **ex)
    for t, w in zip(leaves, want):
        assert np.abs(t.grad.float().cpu().numpy() - w).max() <= 2e-2 * max(1.0, np.abs(w).max())


@pytest.mark.parametrize("cls,shape,heads,dim,bias", [
    (nb.NeighborhoodAttention1D, (130,), 2, 64, True), (nb.NeighborhoodAttention2D, (14, 17), 3, 32, True),
    (nb.NeighborhoodAttention2D, (14, 17), 2, 128, False), (nb.NeighborhoodAttention3D, (6, 9, 11), 2, 64, True)])
def test_layer_as_one_node_matches_the_layer_in_parts(cls, shape, heads, dim, bias):
    """A forward hook sends the layer through its modules one by one: same output, same gradients
    up to the rounding of sums taken in another order (2^-8 of the largest entry: one bf16 step)."""
    torch.manual_seed(43)
    layer = cls(heads * dim, heads, 3, dilation=2, qkv_bias=bias).cuda().bfloat16()
    x, d_y = (torch.randn(2, *shape, heads * dim, device="cuda").bfloat16() for _ in range(2))
    results = []
    for hooked in (False, True):
        handle = layer.qkv.register_forward_hook(lambda *a: None) if hooked else None
        xi = x.clone().requires_grad_()
        y = layer(xi)
        assert ("LayerFunction" in y.grad_fn.name()) != hooked
        results.append([y.detach()] + list(torch.autograd.grad(y, [xi, *layer.parameters()], d_y)))
        with torch.no_grad():
            assert torch.equal(layer(x), y)
        if hooked:
            handle.remove()
    assert L.device_status() == 0
    for a, b in zip(*results):
        assert (a.float() - b.float()).abs().max().item() <= 2 ** -8 * b.float().abs().max().item()


@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 264), (4097, 96), (100352, 384)])
def test_column_sums(rows, cols):
    """fp32 sums rounded once: half a bf16 step (8 significant bits: 2^-8 of the result) plus the fp32
    summation error,
    at most rows 2^-24 of the sum of magnitudes; the same bits twice."""
    torch.manual_seed(47)
    m = torch.randn(rows, cols, device="cuda").bfloat16()
    outs = []
    for _ in range(2):
        out = torch.empty(cols, device="cuda", dtype=torch.bfloat16)
        scratch = torch.empty(L.lib.b200na_column_sum_scratch(rows, cols), device="cuda", dtype=torch.uint8)
        L.check(L.lib.b200na_column_sum(m.data_ptr(), out.data_ptr(), rows, cols, L.BF16,
                                        scratch.data_ptr(), torch.cuda.current_stream().cuda_stream), "")
        outs.append(out)
    want = m.double().sum(0)
    bound = 2 ** -8 * want.abs() + rows * 2 ** -24 * m.double().abs().sum(0)
    assert ((outs[0].double() - want).abs() <= bound * 1.01).all() and torch.equal(*outs)


def test_native_front_leaves_other_calls_to_the_python_front():
    q = torch.randn(1, 12, 12, 2, 64, device="cuda").half()
    for bad in (dict(kernel_size=13), dict(kernel_size=3, stride=4), dict(kernel_size=(3, 3, 3)),
                dict(kernel_size=True), dict(kernel_size=3, is_causal=(1, 0))):
        with pytest.raises(ValueError):
            nb.na2d(q, q, q, **bad)
    with pytest.raises(RuntimeError):
        nb.na2d(q.cpu(), q.cpu(), q.cpu(), 3)
    with pytest.raises(ValueError):
        nb.na2d(q, q, q.float(), 3)
    x = q.clone().requires_grad_()
    (g,) = torch.autograd.grad(nb.na2d(x, q, q, 3).float().sum(), x, create_graph=True)
    with pytest.raises(RuntimeError):
        g.float().sum().backward()


RAGGED = [   # shape, window, stride, dilation, causal, forward (q, kv) tile, backward (q, kv) tile
    ((20, 17), (5, 4), (1, 1), (1, 1), (False, False), (1, 1), (1, 1), (1, 1), (1, 1)),
    ((20, 17), (5, 4), (2, 1), (1, 1), (False, True), (15, 16), (11, 11), (9, 14), (14, 9)),
    ((31, 40), (7, 9), (1, 1), (2, 1), (False, False), (3, 42), (127, 1), (1, 127), (127, 1)),
    ((30, 41), (13, 6), (1, 1), (1, 2), (True, False), (43, 2), (5, 25), (43, 2), (3, 42)),
    ((7, 9, 11), (3, 5, 11), (1, 2, 1), (1, 1, 1), (True, False, False), (7, 3, 6), (7, 3, 6), (7, 3, 6), (5, 5, 5)),
    ((7, 9, 11), (4, 9, 3), (1, 1, 1), (1, 1, 2), (False, False, False), (2, 9, 14), (2, 9, 7), (2, 9, 6), (7, 9, 2)),
    ((300,), (33,), (1,), (3,), (True,), (254,), (101,), (100,), (77,)),
]


@pytest.mark.parametrize("shape,ks,st,di,ca,tq,tkv,bq,bkv", RAGGED)
@pytest.mark.parametrize("D", [64, 128])
def test_tiles_of_any_size(shape, ks, st, di, ca, tq, tkv, bq, bkv, D):
    """Forward and backward with tiles of fewer than 128 tokens, through the C entries for views. What
    shared memory holds from an earlier launch (here: NaN, in tiles of 128 rows) must not matter."""
    torch.manual_seed(53)
    nd, B, Hq, Hkv = len(shape), 2, 4, 2
    q, d_out = (torch.randn(B, *shape, Hq, D, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, *shape, Hkv, D, device="cuda").bfloat16() for _ in range(2))
    out, lse = torch.empty_like(q), torch.empty(q.shape[:-1], device="cuda")
    delta = torch.empty_like(lse)
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    scale, stream = D ** -0.5, torch.cuda.current_stream().cuda_stream
    poison = torch.full((1, 2048, 148, D), float("nan"), device="cuda").bfloat16().requires_grad_()
    geometry = [nd] + [L.ints([int(x) for x in a]) for a in (shape, ks, st, di, ca)]
    sizes = [B, Hq, Hkv, D, L.BF16, scale]
    with torch.no_grad():
        nb.na1d(poison, poison, poison, 512)
    L.check(L.lib.b200na_na_forward_view(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), 0, 0, 0, out.data_ptr(), lse.data_ptr(), *geometry,
        L.ints(tq), L.ints(tkv), *sizes, 0, 0, 0, stream), "b200na_na_forward_view")
    torch.autograd.grad(nb.na1d(poison, poison, poison, 512), poison, poison.detach())
    L.check(L.lib.b200na_na_backward_view(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), d_out.data_ptr(), lse.data_ptr(), 0, 0,
        0, dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), 0, 0, delta.data_ptr(), *geometry, L.ints(bq),
        L.ints(bkv), *sizes, 0, 0, 0, 0, 0, 0, stream), "b200na_na_backward_view")
    assert L.device_status() == 0
    f = [t.float().cpu().numpy() for t in (q, k, v)]
    want_o, want_l = oracle.na_forward(*f, ks, st, di, ca)
    assert np.abs(out.float().cpu().numpy() - want_o).max() <= 2e-2
    assert np.abs(lse.cpu().numpy() - want_l).max() <= 2e-2
    want = oracle.na_backward(*f, d_out.float().cpu().numpy(), ks, st, di, ca)
    for g, w in zip((dq, dk, dv), want):
        assert np.abs(g.float().cpu().numpy() - w).max() <= 2e-2 * max(1.0, np.abs(w).max())


@pytest.mark.parametrize("shape,ks,st,di", [((14, 21, 22), (14, 21, 9), (1, 1, 4), (1, 1, 1)),
                                            ((20, 103), (5, 7), (1, 1), (4, 4)), ((13, 29), (11, 8), (1, 1), (1, 1))])
def test_planned_tiles_8bit(shape, ks, st, di):
    """Shapes whose planned tiles are no powers of two, 8-bit operands: one e4m3 step (1/8)."""
    torch.manual_seed(59)
    q, k, v = (torch.randn(1, *shape, 2, 128).to(torch.float8_e4m3fn) for _ in range(3))
    ca = (False,) * len(shape)
    out = {2: nb.na2d, 3: nb.na3d}[len(shape)](q.cuda(), k.cuda(), v.cuda(), ks, st, di, ca)
    assert L.device_status() == 0
    want, _ = oracle.na_forward(*[t.float().numpy() for t in (q, k, v)], ks, st, di, ca)
    assert np.abs(out.float().cpu().numpy() - want).max() <= 0.125 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("B,nq,nk,hq,hkv,D", [
    (1, 1, 1024, 1, 1, 64),       # two parts of four tiles, the fewest there are
    (2, 3, 16384, 4, 2, 128),     # a decoding step: many parts, GQA
    (1, 130, 5000, 2, 2, 40),     # two query tiles, a ragged last part and tile, a narrow head
    (3, 300, 1537, 3, 1, 128),    # 128-row tiles
    (1, 257, 511, 1, 1, 64),      # too few keys to cut
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dense_attention_over_parts_of_the_keys(B, nq, nk, hq, hkv, D, dtype):
    """Against attention in 64 bits: the result's rounding (2^-8 / 2^-11 of it) and that of the
    probabilities, the same relative size; the registered operator gives the same bits."""
    torch.manual_seed(61)
    q = torch.randn(B, nq, hq, D, device="cuda").to(dtype)
    k, v = (torch.randn(B, nk, hkv, D, device="cuda").to(dtype) for _ in range(2))
    parts = L.lib.b200na_fmha_splits(B, nq, nk, hq, D, L.BF16, 0)
    assert (parts > 1) == (nk >= 1024)
    out, lse = nb.attention(q, k, v, return_lse=True)
    assert L.device_status() == 0
    kd, vd = (t.double().repeat_interleave(hq // hkv, 2) for t in (k, v))
    s = torch.einsum("bqhd,bkhd->bqhk", q.double(), kd) * D ** -0.5
    want = torch.einsum("bqhk,bkhd->bqhd", s.softmax(-1), vd)
    bound = 2 ** (-7 if dtype == torch.bfloat16 else -10) * want.abs().max()
    assert (out.double() - want).abs().max() <= bound
    assert (lse.double() - s.logsumexp(-1)).abs().max() <= 1e-3
    again, lse2 = torch.compile(lambda a, b, c: nb.attention(a, b, c, return_lse=True))(q, k, v)
    assert torch.equal(again, out) and torch.equal(lse2, lse)


FIRST_CALL = """
import sys, threading, torch, natten_b200 as nb
q = torch.randn(1, 24, 40, 2, 128, device="cuda").bfloat16().requires_grad_()
k, v, g = (torch.randn_like(q) for _ in range(3))
pool = [torch.empty(n, device="cuda") for n in (10, 1000, 100000, 1 << 20) for _ in range(8)]
del pool                      # cached memory: nothing below has to ask the driver for any
out = nb.na2d(q, k, v, (7, 9))
torch.cuda.synchronize()
out.backward(g)               # the first GPU work of the engine's thread
want, got = q.grad.clone(), []
def work():                   # the first GPU work of this thread, its backward in the engine's
    got.append(nb.na2d(q, k, v, (7, 9)))
    got.extend(torch.autograd.grad(got[0], q, g))
thread = threading.Thread(target=work)
thread.start(); thread.join()
assert torch.equal(got[0], out) and torch.equal(got[1], want)
print("done")
"""


def test_first_gpu_work_of_a_thread():
    """A thread that has not called the CUDA runtime has no current context, and encoding a tensor map
    needs one."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(nb.__file__)))
    r = subprocess.run([sys.executable, "-c", FIRST_CALL], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "done", r.stderr[-2000:]


def _fresh(t):
    """The same values in standard strides (clone() would keep the odd ones)."""
    return torch.empty(t.shape, dtype=t.dtype, device=t.device).copy_(t)


@pytest.mark.parametrize("op,hq,hkv,D", [("na", 4, 1, 64), ("na", 1, 1, 128), ("na", 1, 1, 40),
                                         ("attention", 4, 1, 64), ("attention", 1, 1, 128)])
def test_one_head_in_heads_first_layout(op, hq, hkv, D):
    """[B, 1, N, D].transpose(1, 2) counts as contiguous, with a head stride that is not D: the same
    results as from standard strides, forward and backward."""
    torch.manual_seed(67)
    q = torch.randn(2, hq, 200, D, device="cuda").bfloat16().transpose(1, 2)
    k, v = (torch.randn(2, hkv, 200, D, device="cuda").bfloat16().transpose(1, 2) for _ in range(2))
    assert k.is_contiguous() and k.stride(2) != D
    d_out = torch.randn(2, 200, hq, D, device="cuda").bfloat16()
    fn = (lambda *a: nb.na1d(*a, 33)) if op == "na" else nb.attention
    results = []
    for leaves in ([q, k, v], [_fresh(t) for t in (q, k, v)]):
        leaves = [t.detach().requires_grad_() for t in leaves]
        out = fn(*leaves)
        assert "NaFunction" in out.grad_fn.name()
        results.append([out.detach(), *torch.autograd.grad(out, leaves, d_out)])
    assert L.device_status() == 0
    for a, b in zip(*results):
        assert torch.equal(a, b)



def _off_16_bytes(t):
    """The same values one element behind a 16-byte boundary, contiguous."""
    u = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape).copy_(t)
    assert u.is_contiguous() and u.data_ptr() % 16
    return u


@pytest.mark.parametrize("case", ["attention", "attention-narrow", "narrow", "folded", "layer"])
def test_output_gradient_off_16_bytes(case):
    """A piece of a flat buffer: autograd passes it on as it is."""
    torch.manual_seed(71)
    if case == "layer":
        layer = nb.NeighborhoodAttention2D(96, 3, 5).cuda().bfloat16()
        x = torch.randn(2, 14, 17, 96, device="cuda").bfloat16().requires_grad_()
        wrt, fn = [x, *layer.parameters()], lambda: layer(x)
    else:
        D = 24 if case in ("narrow", "attention-narrow") else 64
        tokens = (12, 13) if case == "narrow" else (150,)
        wrt = [torch.randn(2, *tokens, 2, D, device="cuda").bfloat16().requires_grad_() for _ in range(3)]
        fn = {"narrow": lambda: nb.na2d(*wrt, 5), "folded": lambda: nb.na1d(*wrt, 9, dilation=5)}.get(
            case, lambda: nb.attention(*wrt))
    d_out = torch.randn_like(fn())
    want = torch.autograd.grad(fn(), wrt, d_out)
    got = torch.autograd.grad(fn(), wrt, _off_16_bytes(d_out))
    assert L.device_status() == 0
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_compiled_backward_with_an_output_gradient_off_16_bytes():
    torch.manual_seed(71)
    wrt = [torch.randn(2, 150, 2, 64, device="cuda").bfloat16().requires_grad_() for _ in range(3)]
    out = torch.compile(nb.attention)(*wrt)
    d_out = torch.randn_like(out)
    want = torch.autograd.grad(out, wrt, d_out, retain_graph=True)
    for a, b in zip(torch.autograd.grad(out, wrt, _off_16_bytes(d_out)), want):
        assert torch.equal(a, b)



@pytest.mark.parametrize("shape,ks,st,di,ca,hq,hkv,D,n_extra", [
    ((150,), (40,), (1,), (1,), (True,), 2, 1, 32, 0), ((150,), (33,), (4,), (3,), (False,), 2, 2, 20, 7),
    ((13, 21), (5, 7), (1, 2), (1, 2), (False, True), 4, 2, 64, 0), ((64,), (64,), (1,), (1,), (True,), 1, 1, 130, 0)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_fp32_non_finite_tokens_stay_inside_their_windows(shape, ks, st, di, ca, hq, hkv, D, n_extra, value):
    """One token of q, k, v or the output gradient is NaN or infinite: the rows that attend it (that it
    attends) are what the oracle makes of them, all others are what they are without it."""
    torch.manual_seed(73)
    fn = {1: nb.na1d, 2: nb.na2d}[len(shape)]
    ops = [torch.randn(1, *shape, h, D) for h in (hq, hkv, hkv, hq)]
    extras = [torch.randn(1, n_extra, hkv, D) for _ in range(2)] if n_extra else []
    for which in range(4):
        for token in (0, 37, 63):
            poisoned = [t.clone() for t in ops]
            poisoned[which].view(-1, ops[which].shape[-2], D)[token, -1, 3] = value
            leaves = [t.cuda().requires_grad_() for t in poisoned[:3]]
            add = dict(zip(("additional_keys", "additional_values"), [t.cuda() for t in extras]))
            out = fn(*leaves, ks, st, di, ca, **add)
            got = [out.detach(), *torch.autograd.grad(out, leaves, poisoned[3].cuda())]
            f = [t.numpy() for t in poisoned]
            ex = dict(add_k=extras[0].numpy(), add_v=extras[1].numpy()) if n_extra else {}
            with np.errstate(invalid="ignore"):
                want = [oracle.na_forward(*f[:3], ks, st, di, ca, **ex)[0],
                        *oracle.na_backward(*f, ks, st, di, ca, **ex)[:3]]
            for g, w in zip(got, want):
                g, on = g.cpu().numpy(), np.isfinite(w)
                assert np.array_equal(np.isfinite(g), on)
                if on.any():    # not where a causal window over everything starts with the token
                    assert np.abs(g[on] - w[on]).max() <= 2e-4 * max(1.0, np.abs(w[on]).max())


@pytest.mark.parametrize("n,win,dil,causal,hq,hkv,D,n_extra", [
    (129, 0, 1, False, 2, 1, 64, 0), (700, 0, 1, True, 3, 3, 128, 0), (1000, 0, 1, False, 2, 2, 40, 0),
    (128, 0, 1, True, 1, 1, 64, 0), (1201, 65, 3, True, 2, 2, 64, 20), (1500, 129, 8, False, 4, 2, 128, 0),
    (4097, 0, 1, True, 1, 1, 64, 0), (4100, 9, 3, True, 2, 2, 64, 40)])
@pytest.mark.parametrize("dtype,size", [(torch.bfloat16, 1.0), (torch.float16, 1.0), (torch.float16, 2.0 ** -10),
                                        (torch.float16, 2.0 ** 10)])
def test_gradients_with_more_bits_than_the_operands(n, win, dil, causal, hq, hkv, D, n_extra, dtype, size):
    """Dense attention and 1-D dilation above 2: P and dS are not rounded to the operands' type. Against
    the CUDA-core kernels, which hold them in fp32: the same up to the results' own rounding. A relative
    difference of 2^-16 (fp16: 2^-20, the sums' order) flips it for 2^-16 / 2^-8 (2^-20 / 2^-11) of the
    entries by 2^-8 (2^-11), 2^-12 (2^-15.5) of the norm where there are thousands of them; with rounded P
    and dS it was 2^-8.6 (2^-11.6)."""
    torch.manual_seed(79)
    q, d_out = (torch.randn(2, n, hq, D, device="cuda").to(dtype) for _ in range(2))
    k, v = (torch.randn(2, n, hkv, D, device="cuda").to(dtype) for _ in range(2))
    d_out = d_out * size
    extras = [torch.randn(2, n_extra, hkv, D, device="cuda").to(dtype) for _ in range(2)] if n_extra else []
    leaves = [t.requires_grad_() for t in [q, k, v] + extras]
    if win:
        add = dict(additional_keys=leaves[3], additional_values=leaves[4]) if n_extra else {}
        out, lse = nb.na1d(*leaves[:3], win, 1, dil, causal, return_lse=True, **add)
    else:
        out, lse = nb.attention(*leaves, is_causal=causal, return_lse=True)
    got = torch.autograd.grad(out, leaves, d_out)
    assert L.device_status() == 0
    with torch.no_grad():
        want = nb.ops.na_backward_simt(q, k, v, out, d_out, lse, *(extras or (None, None)), [win or n], [1],
                                       [dil], [causal], D ** -0.5)
    tol = 2.0 ** -11.5 if dtype == torch.bfloat16 else 2.0 ** -14
    if dtype == torch.float16 and (n if n_extra else win or n) > 4096:
        tol = 0.0                                   # these are the CUDA-core kernels
    for a, b in zip(got, want):
        assert (a.float() - b.float()).norm() <= tol * b.float().norm()


def test_batches_of_more_than_2_to_31_elements():
    """2^20 entries of one query and one key, 32 heads of 128: 2^32 elements. With one key the result is
    its value."""
    B, Hq, D = 1 << 20, 32, 128
    q = torch.zeros(B, 1, Hq, D, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(B, 1, 1, D, device="cuda").bfloat16()
    out = nb.attention(q, v, v)
    for a in range(0, B, B // 8):
        assert torch.equal(out[a:a + B // 8], v[a:a + B // 8].expand(-1, -1, Hq, -1))


def _strided(t):
    """The same values with the axes' strides reversed."""
    return t.permute(*reversed(range(t.dim()))).contiguous().permute(*reversed(range(t.dim())))


@pytest.mark.parametrize("case", ["attention", "na", "na-fp32", "layer", "compiled-attention", "compiled-na"])
def test_saved_tensor_hooks_that_return_other_strides(case):
    torch.manual_seed(83)
    dtype = torch.float32 if case == "na-fp32" else torch.bfloat16
    if case == "layer":
        layer = nb.NeighborhoodAttention2D(96, 3, 5).cuda().bfloat16()
        x = torch.randn(2, 14, 17, 96, device="cuda").bfloat16().requires_grad_()
        wrt, fn = [x, *layer.parameters()], lambda: layer(x)
    else:
        wrt = [torch.randn(2, 12, 13, 2, 64, device="cuda").to(dtype).requires_grad_() for _ in range(3)]
        if "attention" in case:
            wrt = [t.detach().flatten(1, 2).requires_grad_() for t in wrt]
        fn = (lambda: nb.attention(*wrt)) if "attention" in case else (lambda: nb.na2d(*wrt, 5))
        if "compiled" in case:   # the registered operators, as compiled code calls them
            op = nb.functional.ops.fmha_forward if "attention" in case else nb.functional.na_forward_op
            args = (False, 0.125) if "attention" in case else (None, None, [5, 5], [1, 1], [1, 1],
                                                               [False, False], 0.125, [], [], False, [], [])
            fn = lambda: op(*wrt, *args)[0]
    out = fn()
    d_out = torch.randn_like(out)
    want = torch.autograd.grad(out, wrt, d_out)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, _strided):
        out = fn()
    for a, b in zip(torch.autograd.grad(out, wrt, d_out), want):
        assert torch.equal(a, b)


def test_refused_calls_count_no_launches():
    q = _off_16_bytes(torch.randn(1, 12, 12, 2, 64, device="cuda").bfloat16())
    for leaf in (q, q.detach().requires_grad_()):
        before = L.launches
        with pytest.raises(L.NattenB200Error):   # refused by the native front, then by the Python one
            nb.na2d(leaf, q, q, 3)
        assert L.launches == before


@pytest.mark.parametrize("n,win,dil,causal,hq,hkv,D,n_extra", [
    (300, 0, 1, True, 2, 1, 64, 0), (260, 0, 1, True, 2, 2, 40, 0), (700, 33, 3, True, 2, 2, 128, 20),
    (701, 40, 5, False, 4, 2, 64, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_16bit_non_finite_tokens_stay_with_the_rows_that_interact(n, win, dil, causal, hq, hkv, D, n_extra, dtype):
    """Gradients that the CUDA cores computed first: a NaN or an infinity in a key or an output gradient
    reaches the rows that it reached there, and no others."""
    torch.manual_seed(97)
    ops = [torch.randn(2, n, h, D, device="cuda").to(dtype) for h in (hq, hkv, hkv, hq)]
    extras = [torch.randn(2, n_extra, hkv, D, device="cuda").to(dtype) for _ in range(2)] if n_extra else []
    add = dict(zip(("additional_keys", "additional_values"), extras))
    for which, value, token in ((1, float("nan"), 131), (1, float("inf"), 40), (3, float("nan"), 200),
                                (3, float("-inf"), 5), (0, float("nan"), 129)):
        poisoned = [t.clone() for t in ops]
        poisoned[which][1, token, -1, 3] = value
        leaves = [t.requires_grad_() for t in poisoned[:3]]
        if win:
            out, lse = nb.na1d(*leaves, win, 1, dil, causal, return_lse=True, **add)
        else:
            out, lse = nb.attention(*leaves, is_causal=causal, return_lse=True)
        got = torch.autograd.grad(out, leaves, poisoned[3])
        assert L.device_status() == 0
        with torch.no_grad():
            want = nb.ops.na_backward_simt(*poisoned[:3], out, poisoned[3], lse, *(extras or (None, None)),
                                           [win or n], [1], [dil], [causal], D ** -0.5)[:3]
        for a, b in zip(got, want):
            on = b.isfinite()
            assert not on.all() and torch.equal(a.isfinite(), on)
            assert (a[on].float() - b[on].float()).norm() <= 2.0 ** -11.5 * b[on].float().norm()
