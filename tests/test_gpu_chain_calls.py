"""The C calls behind trainable and fp8 layers, where the Python layers never take them: pointers that torch
does not hand out, workspaces with a guard behind them, unusual values."""
import ctypes

import pytest
import torch

import ksmm_b200 as kb
from ksmm_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _train_bytes(pattern_list, batch, code, bs_last):
    sizes = [ctypes.c_size_t() for _ in range(3)]
    pat = _lib.int32_array([v for p in pattern_list for v in p])
    _lib.check(_lib.load().ksmm_cu_chain_train_bytes(len(pattern_list), pat, batch, code, bs_last, *map(ctypes.byref, sizes)))
    return pat, [s.value for s in sizes]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("pattern,batch", [((1, 64, 64, 4), 64), ((4, 64, 64, 4), 64), ((1, 96, 96, 2), 64), ((1, 64, 64, 2), 96),
                                           ((1, 64, 64, 16), 70), ((1, 64, 64, 1), 64)])
@pytest.mark.parametrize("bs_last", [0, 1])
def test_unaligned_input_gradient_stays_inside_the_workspace(pattern, batch, bs_last, dtype):
    """grad_input may start anywhere.  Its kernel is then another one, and where that one would want scratch
    that the workspace does not hold, it runs without.  Tolerance: one rounding step of the type."""
    a, b, c, d = pattern
    code = _lib.KSMM_F32 if dtype == torch.float32 else _lib.KSMM_F16
    pat, (_, _, need) = _train_bytes([pattern], batch, code, bs_last)
    gen = torch.Generator(device=DEV).manual_seed(batch)

    def make(feats):
        return torch.randn((feats, batch) if bs_last else (batch, feats), device=DEV, generator=gen).to(dtype)

    x, g = make(a * c * d), make(a * b * d)
    w = torch.randn(a * d * c, b, device=DEV, generator=gen).to(dtype)
    dense = kb.from_kernel_format_to_dense(w.double(), pattern)
    ref = dense.t() @ (g if bs_last else g.t()).double()
    for shift in (0, 1):
        guard = torch.full((need + (1 << 20),), 0xA5, dtype=torch.uint8, device=DEV)
        gx = torch.full((x.numel() + 64,), 7.0, dtype=dtype, device=DEV)
        gw, gb = torch.empty_like(w), torch.empty(a * b * d, dtype=dtype, device=DEV)
        _lib.check(_lib.load().ksmm_cu_chain_backward(
            x.data_ptr(), (ctypes.c_void_p * 1)(w.data_ptr()), None, None, g.data_ptr(), gx[shift:].data_ptr(),
            (ctypes.c_void_p * 1)(gw.data_ptr()), gb.data_ptr(), guard.data_ptr(), need, batch, 1, pat, code, bs_last, _stream()))
        torch.cuda.synchronize()
        assert bool((guard[need:] == 0xA5).all())
        got = gx[shift:shift + x.numel()].view(x.shape)
        got = (got if bs_last else got.t()).double()
        err = (torch.linalg.norm(got - ref) / torch.linalg.norm(ref)).item()
        assert err < (1e-5 if dtype == torch.float32 else 2.0 ** -11), (shift, err)
        assert bool((gx[:shift] == 7.0).all()) and bool((gx[shift + x.numel():] == 7.0).all())
    kb.check_device()


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_tuning_a_ragged_batch_keeps_the_padded_path(dtype):
    """The copy into padded rows is among the candidates (several times faster at this size); a choice that is
    set for the ragged rows does not reach the padded ones of a chain."""
    pattern, batch = (1, 768, 192, 2), 6501
    lib, code = _lib.load(), _lib.KSMM_F16 if dtype == torch.float16 else _lib.KSMM_F32
    before = kb.default_choice(pattern, batch, dtype, True)
    assert before[2], "this batch is not copied"
    entry = kb.tuner.tune_factor(pattern, batch, dtype, True, nrepeats=5)
    algo, cfg = ctypes.c_int(), ctypes.c_int()
    try:
        assert entry["family"] == "auto" and kb.default_choice(pattern, batch, dtype, True) == before
        assert lib.ksmm_cu_get_choice(batch, *pattern, code, code, 1, ctypes.byref(algo), ctypes.byref(cfg)) != _lib.KSMM_OK
        layer = kb.KSLinear([(6, 64, 64, 1), pattern], dtype=dtype, bs_last=True, device=DEV)
        x = torch.randn(384, batch, device=DEV).to(dtype)
        ref = layer(x)
        _lib.check(lib.ksmm_cu_set_choice(batch, *pattern, code, code, 1, _lib.KSMM_ALGO_SIMT, 2))
        assert torch.equal(layer(x), ref)   # the same kernel, the same bits
    finally:
        lib.ksmm_cu_clear_choice(batch, *pattern, code, code, 1)
    kb.check_device()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -14])
@pytest.mark.parametrize("bs_last", [False, True])
def test_fp8_activations_with_nan_and_infinity(bs_last, scale, dtype):
    """A NaN makes the tensor's scale 1: infinities and large values are then 448 as quantize_e4m3 has it, and
    only the entries that meet the NaN are NaN.  (Identity weights: the results are the quantised inputs.)"""
    n, batch = 64, 48
    layer = kb.KSLinear([(1, n, n, 1)], weights=[torch.eye(n).view(1, n, n, 1)], bias=False, dtype=torch.float8_e4m3fn,
                        bs_last=bs_last, device=DEV)
    x = torch.randn(batch, n, device=DEV).mul_(600 * scale)
    x[3, 5], x[7, 9], x[8, 2] = float("nan"), float("inf"), float("-inf")
    x = (x.t().contiguous() if bs_last else x).to(dtype)
    for clean in (False, True):
        if clean:   # without the NaN the scale is infinite
            x = torch.nan_to_num(x, nan=1.0, posinf=float("inf"), neginf=float("-inf"))
        (wq, sw), = layer._fp8_factors()
        q, s = kb.quantize_e4m3(x)
        ref = kb.forward_fp8(q, wq, bs_last, 1, n, n, 1, s, sw)
        assert torch.equal(torch.isnan(layer(x)), torch.isnan(ref))
        assert torch.equal(torch.nan_to_num(layer(x)), torch.nan_to_num(ref))
    kb.check_device()


@pytest.mark.parametrize("patterns", [[(1, 48, 32, 1)], [(6, 64, 64, 1), (1, 768, 192, 2)]])
@pytest.mark.parametrize("bs_last", [False, True])
def test_bias_gradient_of_long_fp32_batches(patterns, bs_last):
    """A tree over at most 64 neighbours in fp32 (an rms error of 2^-25 per level, about 2^-24 in all), longer sums
    in fp64, one rounding at the end: below 2^-23 of the result's norm at any length."""
    layer = kb.KSLinear(patterns, dtype=torch.float32, bs_last=bs_last, device=DEV, requires_grad=True)
    for batch in (640, 50176, 50177):
        x = torch.zeros((layer.in_size, batch) if bs_last else (batch, layer.in_size), device=DEV)
        gen = torch.Generator(device=DEV).manual_seed(batch)
        g = torch.randn((layer.out_size, batch) if bs_last else (batch, layer.out_size), device=DEV, generator=gen)
        for want_x in (False, True):
            layer.bias.grad = None
            layer(x.requires_grad_(want_x)).backward(g)
            ref = g.double().sum(1 if bs_last else 0)
            err = torch.linalg.norm(layer.bias.grad.reshape(-1).double() - ref) / torch.linalg.norm(ref)
            assert err.item() < 2.0 ** -23, (batch, want_x, err.item())
    kb.check_device()


@pytest.mark.parametrize("bs_last", [False, True])
@pytest.mark.parametrize("patterns", [[(1, 64, 64, 16), (4, 64, 64, 4), (16, 64, 64, 1)], [(6, 64, 64, 1), (1, 768, 192, 2)],
                                      [(1, 192, 768, 4), (4, 192, 192, 1)]])
def test_trainable_fp32_layers_keep_their_precision(patterns, bs_last):
    """Against fp64, the layer's result and its input's gradient are no further off than one factor after the
    other (a tenth more at most: the same sums may run in another order)."""
    layer = kb.KSLinear(patterns, dtype=torch.float32, bs_last=bs_last, bias=False, device=DEV, requires_grad=True)
    dense = [kb.from_kernel_format_to_dense(f.data.double(), p) for f, p in zip(layer.factors, patterns)]
    for batch in (100, 640, 1001):
        gen = torch.Generator(device=DEV).manual_seed(batch)
        x = torch.randn((layer.in_size, batch) if bs_last else (batch, layer.in_size), device=DEV, generator=gen)
        g = torch.randn((layer.out_size, batch) if bs_last else (batch, layer.out_size), device=DEV, generator=gen)
        y64, x64 = (x if bs_last else x.t()).double(), (g if bs_last else g.t()).double()
        for m in dense:
            y64 = m @ y64
        for m in reversed(dense):
            x64 = m.t() @ x64

        def errors(run):
            xi = x.clone().requires_grad_(True)
            y = run(xi)
            y.backward(g)
            return [(torch.linalg.norm((v if bs_last else v.t()).double() - r) / torch.linalg.norm(r)).item()
                    for v, r in ((y.detach(), y64), (xi.grad, x64))]

        def one_by_one(y):
            for p, f in zip(patterns, layer.factors):
                y = kb.FactorFunction.apply(y, f, bs_last, *p)
            return y

        for name, new, old in zip(("y", "x"), errors(layer), errors(one_by_one)):
            assert new < 1.1 * old, (name, batch, new, old)
    kb.check_device()


def test_fp8_layer_of_more_factors_than_one_call_takes():
    """65 factors run one by one; with 64 of them both ways agree."""
    n = 16
    for count in (64, 65):
        layer = kb.KSLinear([(1, n, n, 1)] * count, weights=[torch.eye(n).view(1, n, n, 1)] * count, bias=False,
                            dtype=torch.float8_e4m3fn, device=DEV)
        x = torch.randn(8, n, device=DEV, dtype=torch.bfloat16)
        y = x
        for wq, sw in layer._fp8_factors():
            q, s = kb.quantize_e4m3(y)
            y = kb.forward_fp8(q, wq, False, 1, n, n, 1, s, sw)
        assert torch.equal(layer(x), y)
    kb.check_device()


def _weight_gradient(x, g, bs_last, pattern, fallback=False):
    """ksmm_cu_backward_weights; without a workspace it runs on the FFMA kernel."""
    a, b, c, d = pattern
    lib, code = _lib.load(), {torch.float32: _lib.KSMM_F32, torch.float16: _lib.KSMM_F16, torch.bfloat16: _lib.KSMM_BF16}[x.dtype]
    batch = x.shape[1] if bs_last else x.shape[0]
    need = 0 if fallback else lib.ksmm_cu_backward_weights_workspace_bytes(batch, a, b, c, d, code, int(bs_last))
    ws, out = torch.empty(max(need, 1), dtype=torch.uint8, device=DEV), torch.empty(a * c * d, b, dtype=x.dtype, device=DEV)
    _lib.check(lib.ksmm_cu_backward_weights(x.data_ptr(), g.data_ptr(), out.data_ptr(), ws.data_ptr() if need else None, need,
                                            batch, a, b, c, d, code, int(bs_last), _stream()))
    return out


@pytest.mark.parametrize("bs_last", [False, True])
@pytest.mark.parametrize("pattern", [(1, 64, 64, 1), (2, 64, 32, 2), (1, 50, 70, 3), (1, 41, 37, 1)])
def test_fp32_weight_gradients_of_infinite_operands(pattern, bs_last):
    """Infinities, NaN and sums past the largest float are what the FFMA kernel makes of them, bit for bit; the
    other sums are those of the finite operands."""
    a, b, c, d = pattern
    for batch in (128, 1001):
        gen = torch.Generator(device=DEV).manual_seed(batch)
        x = torch.randn(a * c * d, batch, device=DEV, generator=gen)
        g = torch.randn(a * b * d, batch, device=DEV, generator=gen)
        g[10, batch - 1] = 0.0
        finite = _weight_gradient(*((x, g) if bs_last else (x.t().contiguous(), g.t().contiguous())), bs_last, pattern)
        inf = float("inf")
        x[3, 5], x[7, batch - 1], x[11, 40], x[12, 3] = inf, -inf, 3.4e38, float("nan")
        g[2, 9], g[8, 0], g[9, 40] = -inf, inf, -3e38
        x, g = (x, g) if bs_last else (x.t().contiguous(), g.t().contiguous())
        dw, ref = (_weight_gradient(x, g, bs_last, pattern, fallback=f) for f in (False, True))
        odd = ~torch.isfinite(ref)
        assert odd.any() and torch.isinf(ref).any() and not odd.all()
        assert torch.equal(torch.isfinite(dw), ~odd)
        assert torch.equal(torch.nan_to_num(dw[odd], nan=7.0), torch.nan_to_num(ref[odd], nan=7.0))
        same = ~odd & torch.isfinite(finite) & (ref.abs() < 1e30)
        assert (torch.linalg.norm((dw - finite)[same]) / torch.linalg.norm(finite[same])).item() < 1e-5
    kb.check_device()


@pytest.mark.parametrize("bs_last", [False, True])
@pytest.mark.parametrize("pattern", [(1, 64, 64, 1), (2, 96, 160, 2), (1, 50, 70, 3)])
def test_fp32_weight_gradients_of_a_few_entries(pattern, bs_last):
    """Masked batches, against 64 bits and the FFMA kernel.  One entry is one product, rounded once, 2^-24, after the
    split has left out two terms of at most 2^-25: as the FMA has it.  m entries in different splits of the batch
    round every term and every sum, 2 m - 1 times where a chain of FMAs rounds m times: below sqrt(2) times its
    error.  Dense batches are closer than the chain."""
    a, b, c, d = pattern
    for batch in (128, 1001, 6272):
        for count in (1, 2, 3, 4, 16, 64, batch):
            gen = torch.Generator(device=DEV).manual_seed(batch + count)
            x = torch.randn(a * c * d, batch, device=DEV, generator=gen)
            g = torch.randn(a * b * d, batch, device=DEV, generator=gen)
            g[:, torch.randperm(batch, device=DEV, generator=gen)[count:]] = 0
            ref = torch.einsum("ikln,ijln->ilkj", x.double().reshape(a, c, d, batch), g.double().reshape(a, b, d, batch))
            ref = ref.reshape(a * d * c, b)
            x, g = (x, g) if bs_last else (x.t().contiguous(), g.t().contiguous())
            off = [_weight_gradient(x, g, bs_last, pattern, fallback=f).double() - ref for f in (False, True)]
            new, old = (torch.linalg.norm(o).item() for o in off)
            assert new < {1: 1.05, batch: 1.0}.get(count, 2 ** 0.5) * old, (batch, count, new, old)
            if count == 1:
                assert (off[0].abs() / ref.abs()).max().item() < 2.0 ** -23
    kb.check_device()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("d", [2, 4])
def test_weight_gradient_of_a_block_ordered_intermediate(d, dtype):
    """Layout 2 of ksmm_cu_chain_backward, also where no forward of that type keeps it: every block of the factor is
    read.  Tolerance: one rounding step of the type (fp32: its sums)."""
    pats, batch = [(2, 32 * d, 64, 1), (1, 96, 64, d)], 200
    gen = torch.Generator(device=DEV).manual_seed(d)
    code = _lib.KSMM_F32 if dtype == torch.float32 else _lib.KSMM_F16
    pat, (saved_bytes, _, need) = _train_bytes(pats, batch, code, 0)
    x, h, g = (torch.randn(batch, n, device=DEV, generator=gen).to(dtype) for n in (128, 64 * d, 96 * d))
    w = [torch.randn(a * c * q, b, device=DEV, generator=gen).to(dtype) for a, b, c, q in pats]
    saved = torch.zeros(saved_bytes, dtype=torch.uint8, device=DEV)
    saved.view(dtype)[:h.numel()] = h.view(batch, 64, d).transpose(1, 2).reshape(-1)
    gw, ws = torch.empty_like(w[1]), torch.empty(need, dtype=torch.uint8, device=DEV)
    _lib.check(_lib.load().ksmm_cu_chain_backward(
        x.data_ptr(), (ctypes.c_void_p * 2)(*[v.data_ptr() for v in w]), saved.data_ptr(), (ctypes.c_int32 * 1)(2), g.data_ptr(), None,
        (ctypes.c_void_p * 2)(None, gw.data_ptr()), None, ws.data_ptr(), need, batch, 2, pat, code, 0, _stream()))
    ref = torch.einsum("nkl,njl->lkj", h.double().view(batch, 64, d), g.double().view(batch, 96, d)).reshape(64 * d, 96)
    err = (torch.linalg.norm(gw.double() - ref) / torch.linalg.norm(ref)).item()
    assert err < (1e-6 if dtype == torch.float32 else 2.0 ** -11), err
    kb.check_device()


@pytest.mark.parametrize("native", [True, False])
def test_training_raises_library_statuses(native, monkeypatch):
    """A status in the backward (fp32 batches this short take at most 65535 blocks) is a KsmmError with that status,
    through the extension module as through ctypes."""
    from ksmm_b200 import kernel as kk
    if not native:
        monkeypatch.setattr(kk, "_native", None)
    layer = kb.KSLinear([(65536, 1, 1, 1)], dtype=torch.float32, bias=False, device=DEV, requires_grad=True)
    x = torch.randn(2, 65536, device=DEV, requires_grad=True)
    y = layer(x)
    assert torch.equal(y.detach(), x.detach() * layer.factors[0].detach().reshape(-1))
    with pytest.raises(kb.KsmmError) as err:
        y.sum().backward()
    assert err.value.status == _lib.KSMM_ERR_UNSUPPORTED and "blocks" in str(err.value)
    kb.check_device()


@pytest.mark.parametrize("bs_last", [False, True])
def test_trainable_layers_with_another_bias(bs_last):
    """A bias of another type or with strides is added outside the node, as torch promotes it."""
    layer = kb.KSLinear([(4, 48, 48, 1), (1, 192, 48, 4)], dtype=torch.float16, bs_last=bs_last, device=DEV, requires_grad=True)
    x = torch.randn((192, 40) if bs_last else (40, 192), device=DEV, dtype=torch.float16)
    shape = layer.bias.shape
    with torch.no_grad():
        plain = layer(x) - layer.bias.detach().reshape((-1, 1) if bs_last else (1, -1))
    for bias in (torch.randn(768, device=DEV), torch.randn(768, 2, device=DEV, dtype=torch.float16)[:, 0]):
        layer.bias = torch.nn.Parameter(bias.view(shape) if bias.is_contiguous() else bias)
        y = layer(x)
        want = plain.float() + bias.float().reshape((-1, 1) if bs_last else (1, -1))
        assert y.dtype == torch.promote_types(torch.float16, bias.dtype)
        assert (torch.linalg.norm(y.float() - want) / torch.linalg.norm(want)).item() < 2.0 ** -10
        y.float().sum().backward()
        assert torch.equal(layer.bias.grad.float(), torch.full_like(layer.bias.grad, 40.0).float())
        layer.zero_grad(set_to_none=True)
    kb.check_device()


@pytest.mark.parametrize("patterns,dtype,batch,turn", [
    ([(4, 40, 33, 16), (1, 72, 160, 16)], torch.bfloat16, 128, False), ([(3, 48, 192, 2), (1, 136, 48, 6)], torch.bfloat16, 1024, False),
    ([(3, 72, 136, 4), (1, 64, 216, 4)], torch.float32, 256, False), ([(1, 100, 128, 4)], torch.float32, 300, True),
    ([(4, 32, 40, 4)], torch.float16, 64, True), ([(2, 40, 17, 8)], torch.bfloat16, 129, True), ([(2, 64, 64, 1)], torch.float16, 64, True)])
def test_layers_take_inputs_that_start_anywhere(patterns, dtype, batch, turn):
    """Layers whose chain has a region for transposed copies, on a view that starts off a 16-byte boundary: the
    first factor's kernel is another one, with other scratch.  Tolerance: one rounding step per factor (fp32: its
    sums)."""
    layer = kb.KSLinear(patterns, dtype=dtype, bs_last=False, out_bs_last=turn, device=DEV)
    buf = torch.randn(batch * layer.in_size + 8, device=DEV).to(dtype)
    step = {torch.float32: 2.0 ** -19, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    for shift in (0, 1, 2):
        x = buf[shift:shift + batch * layer.in_size].view(batch, layer.in_size)
        with torch.no_grad():
            y = layer(x)
        ref = x.double()
        for f, p in zip(layer.factors, patterns):
            ref = ref @ kb.from_kernel_format_to_dense(f.data.double(), p).t()
        ref = ref + layer.bias.double().reshape(1, -1)
        err = (torch.linalg.norm((y.t() if turn else y).double() - ref) / torch.linalg.norm(ref)).item()
        assert err < step * len(patterns), (shift, err)
    kb.check_device()


@pytest.mark.parametrize("bs_last", [False, True])
def test_trainable_layers_with_one_bias_for_all_outputs(bs_last):
    """A bias of one element is added to every output, and its gradient is the sum over all of them."""
    layer = kb.KSLinear([(4, 48, 48, 1), (1, 192, 48, 4)], dtype=torch.float32, bs_last=bs_last, device=DEV, requires_grad=True)
    x = torch.randn((192, 40) if bs_last else (40, 192), device=DEV)
    layer.bias = torch.nn.Parameter(torch.zeros(1, device=DEV))
    plain = layer(x).detach()
    layer.bias = torch.nn.Parameter(torch.full((1,), 0.5, device=DEV))
    y = layer(x)
    assert torch.equal(y.detach(), plain + 0.5)
    y.sum().backward()
    assert layer.bias.grad.item() == 768 * 40
    kb.check_device()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("patterns", [[(4, 192, 192, 1), (1, 192, 192, 4)], [(2, 64, 40, 1), (1, 72, 32, 4)],
                                      [(2, 128, 64, 1), (2, 136, 64, 2)]])
def test_grouped_block_ordered_chains(patterns, dtype):
    """One launch per factor for all groups, each group with its own weights and bias, at batches that end inside a
    tile.  Tolerance: two factors, one rounding step each."""
    gen = torch.Generator(device=DEV).manual_seed(7)
    group = kb.KSLinearGroup([kb.KSLinear(patterns, dtype=dtype, device=DEV) for _ in range(3)])
    for batch in (1, 33, 197, 1001):
        x = torch.randn(batch, group.layers[0].in_size, device=DEV, generator=gen).to(dtype)
        group(x)
        before = kb.launch_count()
        out = group(x)
        assert kb.launch_count() - before == len(patterns), batch
        for y, layer in zip(out, group.layers):
            ref = x.double()
            for f, p in zip(layer.factors, patterns):
                ref = ref @ kb.from_kernel_format_to_dense(f.data.double(), p).t()
            ref = ref + layer.bias.double()
            err = (torch.linalg.norm(y.double() - ref) / torch.linalg.norm(ref)).item()
            assert err < (2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7), (batch, err)
    kb.check_device()
