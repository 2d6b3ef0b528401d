"""The drop-in boundary: import paths and Function protocol of the reference (main.py:2-6;
universal_attention_autograd.py:9, :41-44, :104, :166-169; Universal_Attention/universal_attention.py:7, :27-31)."""
import inspect

import pytest
import torch


def _classes():
    from universal_attention_autograd import SMVecMatMul, UniversalAttention, UniversalAttention2
    from Universal_Attention.universal_attention import UniversalAttention as KernelUA
    return UniversalAttention, UniversalAttention2, KernelUA, SMVecMatMul


def test_reference_import_paths_resolve_to_the_cuda_backed_classes():
    import universal_attention_triton_b200 as pkg
    ua1, ua2, kua, smv = _classes()
    assert ua1 is pkg.UniversalAttention and ua2 is pkg.UniversalAttention2 and smv is pkg.SMVecMatMul
    from universal_attention_triton_b200.Universal_Attention.universal_attention import UniversalAttention as inner
    assert kua is inner


def test_functions_follow_the_new_style_protocol():
    for cls in _classes()[:3]:
        params = list(inspect.signature(cls.forward).parameters)
        assert params == ["kc", "vc", "xq", "static_src", "static_dest"], params      # no ctx
        assert list(inspect.signature(cls.setup_context).parameters) == ["ctx", "inputs", "outputs"]
        assert "setup_context" in cls.__dict__ and "backward" in cls.__dict__
    smv = _classes()[3]
    assert list(inspect.signature(smv.forward).parameters) == ["mat", "vec"]


def test_note_on_gradients_that_vanish_before_each_chunk():
    """The note SMVecMatMul.backward leaves on its results (the native nodes' registry; no GPU): it holds the tensor's version counter,
    an in-place change voids it, and tensors that autograd derives (a sum of two gradients, a hook's replacement) do not carry
    it -- so the operator's backward falls back to the full path whenever the zeros are not guaranteed."""
    from universal_attention_triton_b200 import universal_attention_autograd as M
    g = torch.zeros(2, 3)
    assert not M._masked_zero(g)
    M._mark_masked_zero(g)
    assert M._masked_zero(g)
    assert not M._masked_zero(g + 0)             # a new tensor
    assert not M._masked_zero(g.clone())
    g.add_(1.0)                                  # in-place change: the note is void
    assert not M._masked_zero(g)

    # through autograd: the note reaches the next node only when the tensor itself is handed on
    seen = []

    class Probe(torch.autograd.Function):
        @staticmethod
        def forward(x):
            return x * 1.0

        @staticmethod
        def setup_context(ctx, inputs, output):
            pass

        @staticmethod
        def backward(ctx, g):
            seen.append(M._masked_zero(g))
            return g

    class Source(torch.autograd.Function):
        @staticmethod
        def forward(x):
            return x.sum()

        @staticmethod
        def setup_context(ctx, inputs, output):
            ctx.shape = inputs[0].shape

        @staticmethod
        def backward(ctx, g):
            out = torch.ones(ctx.shape) * g
            M._mark_masked_zero(out)
            return out

    x = torch.randn(4, requires_grad=True)
    Source.apply(Probe.apply(x)).backward()                                  # single consumer: handed on
    y = Probe.apply(x)
    (Source.apply(y) + y.sum()).backward()                                   # two consumers: autograd sums the gradients
    y = Probe.apply(x)
    y.register_hook(lambda g: g * 1.0)                                       # a hook replaces the tensor
    Source.apply(y).backward()
    assert seen == [True, False, False]


def test_cpu_tensors_are_refused_not_computed():
    ua1 = _classes()[0]
    b, h, r, n, c, d = 1, 1, 1, 2, 16, 8
    args = (torch.randn(b, h, n, c, d), torch.randn(b, h, n, c, d), torch.randn(b, h, r, n * c, d),
            torch.rand(b, h, n, c), torch.rand(b, h, n * c))
    with pytest.raises(RuntimeError, match="no CPU path"):
        ua1.apply(*args)


def _cpu_args():
    b, h, r, n, c, d = 1, 1, 1, 2, 16, 8
    return (torch.randn(b, h, n, c, d), torch.randn(b, h, n, c, d), torch.randn(b, h, r, n * c, d),
            torch.rand(b, h, n, c), torch.rand(b, h, n * c))


def test_a_subclass_runs_its_own_forward_and_backward():
    """``apply`` of a subclass takes the Function protocol, with whatever the subclass overrides (host logic, no GPU)."""
    for base in _classes()[:3]:
        class Mine(base):
            @staticmethod
            def forward(kc, vc, xq, static_src, static_dest):
                return kc.sum() + 0, vc * 3

            @staticmethod
            def setup_context(ctx, inputs, outputs):
                ctx.save_for_backward(*inputs)

            @staticmethod
            def backward(ctx, g_out, g_denom):
                kc = ctx.saved_tensors[0]
                return g_out * torch.ones_like(kc), g_denom * 3, None, None, None

        args = _cpu_args()
        kc, vc = args[0].requires_grad_(), args[1].requires_grad_()
        out, denom = Mine.apply(*args)
        assert torch.equal(denom, vc * 3) and out.shape == ()
        gk, gv = torch.autograd.grad([out, denom], [kc, vc], [torch.tensor(2.0), torch.ones_like(vc)])
        assert torch.equal(gk, torch.full_like(kc, 2.0)) and torch.equal(gv, torch.full_like(vc, 3.0))

    class Last(_classes()[3]):
        @staticmethod
        def forward(mat, vec):
            return mat[..., -1] * 1.0
    assert Last.apply(torch.randn(1, 1, 1, 4, 2, 3), torch.randn(1, 1, 1, 4, 3)).shape == (1, 1, 1, 4, 2)


def test_forward_mode_is_refused_not_dropped(monkeypatch):
    """The Functions have no forward-mode formula: a dual input raises in eager mode too (a native node would return results
    without a tangent); a forward-mode level without dual inputs changes nothing."""
    import torch.autograd.forward_ad as fwad
    from universal_attention_triton_b200 import universal_attention_autograd as M
    monkeypatch.setattr(M, "_forward", lambda kc, vc, xq, ss, sd: (kc * 1.0, vc * 1.0))
    ua1 = _classes()[0]
    args = _cpu_args()
    with fwad.dual_level():
        assert torch.equal(ua1.apply(*args)[0], args[0])
        with pytest.raises(RuntimeError, match="forward AD|jvp"):
            ua1.apply(fwad.make_dual(args[0], torch.ones_like(args[0])), *args[1:])


def test_shape_asserts_fire_like_the_reference():
    ua1, ua2, kua, _ = _classes()
    b, h, r, n, c, d = 1, 1, 1, 2, 16, 8
    kc = torch.randn(b, h, n, c, d)
    with pytest.raises(AssertionError):
        ua1.apply(kc, kc, torch.randn(b, h, r, n * c, d), torch.rand(b, h, n, c), torch.rand(b, h, n * c + 1))
    with pytest.raises(AssertionError):
        kua.apply(kc, kc[:, :, :1], torch.randn(b, h, r, n, c, d), torch.rand(b, h, n, c), torch.rand(b, h, n, c))


@pytest.mark.gpu
def test_reference_driver_flow_through_the_import_shims():
    """main.py:41-62 with the reference's own import lines: clone().requires_grad_(), SMVecMatMul, retain_grad on the
    two outputs, pow(2).sum().backward(); all three entry points against the oracle on the driver's rand inputs."""
    from oracle import ua_oracle as O
    from tests._util import rel_fro
    ua1, ua2, kua, smv = _classes()
    b, s, n_kv, rep, d, c = 2, 256, 2, 2, 64, 64
    n_c = s // c
    g = torch.Generator().manual_seed(3)
    q = torch.rand(b, s, n_kv * rep, d, generator=g)
    k = torch.rand(b, s, n_kv, d, generator=g)
    v = torch.rand(b, s, n_kv, d, generator=g)
    st = torch.rand(b, s, 2 * n_kv, generator=g)
    xq = q.transpose(1, 2).reshape(b, n_kv, rep, s, d)
    kc = k.transpose(1, 2).reshape(b, n_kv, n_c, c, d)
    vc = v.transpose(1, 2).reshape(b, n_kv, n_c, c, d)
    st = st.view(b, s, 2, n_kv).permute(2, 0, 3, 1)
    ss, sd = st[0].reshape(b, n_kv, n_c, c), st[1].reshape(b, n_kv, s)
    _, merged_ref, _, _, grads_ref = O.driver_step(kc, vc, xq, ss, sd)
    ref = dict(zip(("dkc", "dvc", "dxq", "dsrc", "ddest"), grads_ref), merged=merged_ref)
    for fn, two_d in ((ua1, False), (ua2, True), (kua, True)):
        kc_, vc_, ss_ = (t.clone().detach().cuda().requires_grad_() for t in (kc, vc, ss))
        if two_d:
            xq_ = xq.view(b, n_kv, rep, n_c, c, d).clone().detach().cuda().requires_grad_()
            sd_ = sd.view(b, n_kv, n_c, c).clone().detach().cuda().requires_grad_()
        else:
            xq_, sd_ = xq.clone().detach().cuda().requires_grad_(), sd.clone().detach().cuda().requires_grad_()
        output, denom = fn.apply(kc_, vc_, xq_, ss_, sd_)
        out = smv.apply(output, denom)
        output.retain_grad()
        denom.retain_grad()
        out.pow(2).sum().backward()
        assert output.grad is not None and denom.grad is not None
        assert (out.cpu().reshape(ref["merged"].shape) - ref["merged"]).abs().max().item() <= 1e-4
        for name, t in (("dkc", kc_), ("dvc", vc_), ("dxq", xq_), ("dsrc", ss_), ("ddest", sd_)):
            assert rel_fro(t.grad.cpu().reshape(ref[name].shape), ref[name]) <= 1e-4, (fn, name)


@pytest.mark.gpu
def test_backward_recomputes_when_only_the_inputs_were_saved():
    """torch.func.grad drives forward / setup_context with its own wrappers; the Function must also work when the
    forward's by-products did not reach setup_context (they are then recomputed)."""
    from oracle import ua_oracle as O
    from tests._util import rel_fro
    from universal_attention_triton_b200 import universal_attention_autograd as M
    ua1, _, _, smv = _classes()
    ins = O.make_inputs(1, 1, 2, 256, 64, 64, dtype=torch.float32, seed=5)
    ref = dict(zip(("dkc", "dvc", "dxq", "dsrc", "ddest"), O.driver_step(*ins)[4]))

    def loss(kc, vc, xq, ss, sd):
        return smv.apply(*ua1.apply(kc, vc, xq, ss, sd)).pow(2).sum()

    grads = torch.func.grad(loss, argnums=(0, 1, 2, 3, 4))(*[t.cuda() for t in ins])
    for name, gr in zip(("dkc", "dvc", "dxq", "dsrc", "ddest"), grads):
        assert rel_fro(gr.cpu(), ref[name]) <= 1e-4, name

    class Ctx:           # setup_context without the by-products: a plain 2-tuple of fresh tensors
        def save_for_backward(self, *ts):
            self.saved_tensors = ts
    xs = [t.cuda() for t in ins]
    out, denom = M._forward(*xs)
    ctx = Ctx()
    M._setup_context(ctx, tuple(xs), (out.clone(), denom.clone()))
    assert not ctx.ua_has_extras and len(ctx.saved_tensors) == 5
    g_out = torch.randn_like(out)
    g_denom = torch.randn_like(denom)
    got = M._backward(ctx, g_out, g_denom)
    want = O.ua_backward(*ins, g_out.cpu(), g_denom.cpu())
    for a, b_, name in zip(got, want, ("dkc", "dvc", "dxq", "dsrc", "ddest")):
        assert rel_fro(a.cpu(), b_) <= 1e-4, name


@pytest.mark.gpu
def test_own_output_is_saved_for_backward_unless_switched_off():
    """By default the Functions save their own output with the inputs (the tensor-core backward takes the row term of the
    softmax gradient from out . g_out); switched off, they save the reference's five inputs plus the two by-products.
    Same gradients either way, up to the rounding of the bf16 output."""
    import universal_attention_triton_b200 as ua
    from oracle import ua_oracle as O
    from tests._util import rel_fro
    from universal_attention_triton_b200 import universal_attention_autograd as M
    ins = O.make_inputs(1, 2, 2, 512, 128, 64, dtype=torch.bfloat16, seed=9)

    class Ctx:
        def save_for_backward(self, *ts):
            self.saved_tensors = ts
    results = {}
    try:
        for on in (True, False):
            ua.set_save_output(on)
            xs = [t.cuda() for t in ins]
            out, denom = M._forward(*xs)
            ctx = Ctx()
            M._setup_context(ctx, tuple(xs), (out, denom))
            assert ctx.ua_has_extras and ctx.ua_has_out == on
            assert (ctx.saved_tensors[-1] is out) == on
            gen = torch.Generator(device="cuda").manual_seed(11)
            g_out = torch.randn(out.shape, generator=gen, device="cuda").to(out.dtype)
            g_denom = torch.randn(denom.shape, generator=gen, device="cuda")
            results[on] = [t.float().cpu() for t in M._backward(ctx, g_out, g_denom)]
    finally:
        ua.set_save_output(True)
    for a, b_, name in zip(results[True], results[False], ("dkc", "dvc", "dxq", "dsrc", "ddest")):
        assert torch.isfinite(a).all() and rel_fro(a, b_) <= 2e-2, (name, rel_fro(a, b_))


@pytest.mark.gpu
def test_error_of_a_backward_reaches_the_caller_with_its_type():
    """A call that the library refuses on the host (here: an upstream gradient off its 16-byte boundary) raises UaLibraryError from
    the engine's thread too, with the library's message."""
    from oracle import ua_oracle as O
    from universal_attention_triton_b200 import ops
    from universal_attention_triton_b200._lib import UaLibraryError
    ua1 = _classes()[0]
    xs = [t.cuda().requires_grad_() for t in O.make_inputs(1, 1, 1, 256, 128, 64, dtype=torch.bfloat16, seed=3)]
    out, denom = ua1.apply(*xs)
    shifted = torch.zeros(out.numel() + 1, dtype=out.dtype, device="cuda")[1:].view(1, 1, 2, 1, 256, 64)
    with pytest.raises(UaLibraryError, match="ua_bwd failed"):
        torch.autograd.grad([out, denom], xs, [ops.as_reference_out(shifted), torch.zeros_like(denom)])


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["two_consumers", "in_place_hook"])
def test_gradients_before_each_chunk_that_join_the_merges_are_not_lost(how):
    """In the native graph: a gradient of the operator's outputs that is more than SMVecMatMul's -- the sum with another
    consumer's (which autograd may form in place, in the noted tensor), or an in-place change by a hook -- takes the full path.
    Against the oracle on the gradients that really arrive, with most of their norm on the rows before the chunks."""
    import universal_attention_triton_b200 as ua
    from oracle import ua_oracle as O
    from tests._util import rel_fro, valid_row_mask
    b, h, r, L, c, d = 1, 2, 2, 512, 128, 64
    n = L // c
    ins = O.make_inputs(b, h, r, L, c, d, dtype=torch.bfloat16, seed=12)
    gen = torch.Generator().manual_seed(2)
    before = ~valid_row_mask(L, n, c)
    extra = (torch.randn(b, h, r, L, d, n, generator=gen) * before.view(L, 1, n)).bfloat16().cuda()
    extra_den = (torch.randn(b, h, r, L, n, generator=gen) * before).bfloat16().cuda()
    xs = [t.cuda().requires_grad_() for t in ins]
    out, denom = ua.UniversalAttention.apply(*xs)
    arrived = []
    if how == "two_consumers":
        out.register_hook(lambda g: arrived.append(g.clone()))
        denom.register_hook(lambda g: arrived.append(g.clone()))
        loss = ua.SMVecMatMul.apply(out, denom).float().sum() + (out * extra).sum() + (denom * extra_den).sum()
    else:
        out.register_hook(lambda g: arrived.append(g.add_(extra).clone()) and None)
        denom.register_hook(lambda g: arrived.append(g.add_(extra_den).clone()) and None)
        loss = ua.SMVecMatMul.apply(out, denom).float().sum()
    grads = torch.autograd.grad(loss, xs)
    g_out = next(t for t in arrived if t.dim() == 6).float().cpu()
    g_den = next(t for t in arrived if t.dim() == 5).float().cpu()
    assert (g_out * before.view(L, 1, n)).norm() > 0.5 * extra.float().norm().cpu()
    for got, want, name in zip(grads, O.ua_backward(*[t.float() for t in ins], g_out, g_den), ("dkc", "dvc", "dxq", "dsrc", "ddest")):
        assert rel_fro(got.float().cpu(), want) <= 5e-2, (name, rel_fro(got.float().cpu(), want))


@pytest.mark.gpu
def test_native_node_saves_its_output_unless_switched_off():
    """The eager path (a native node): which tensors it saves under either setting of ``set_save_output``, that an in-place change of
    a saved output is noticed, and that both settings give the gradients of the oracle."""
    import universal_attention_triton_b200 as ua
    from oracle import ua_oracle as O
    from tests._util import rel_fro
    ins = O.make_inputs(1, 2, 2, 512, 128, 64, dtype=torch.bfloat16, seed=9)
    gen = torch.Generator(device="cuda").manual_seed(11)
    try:
        for on in (True, False):
            ua.set_save_output(on)
            xs = [t.cuda().requires_grad_() for t in ins]
            packed = []
            with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(tuple(t.shape)) or t, lambda t: t):
                out, denom = ua.UniversalAttention.apply(*xs)
            assert packed.count(tuple(out.shape)) == int(on), packed
            for x in xs:
                assert tuple(x.shape) in packed
            g_out = torch.randn(out.shape, generator=gen, device="cuda").to(out.dtype)
            g_den = torch.randn(denom.shape, generator=gen, device="cuda").to(denom.dtype)
            want = O.ua_backward(*[t.float() for t in ins], g_out.float().cpu(), g_den.float().cpu())
            for got, ref, name in zip(torch.autograd.grad([out, denom], xs, [g_out, g_den]), want, ("dkc", "dvc", "dxq", "dsrc", "ddest")):
                assert rel_fro(got.float().cpu(), ref) <= 5e-2, (on, name)
            out, denom = ua.UniversalAttention.apply(*xs)
            with torch.no_grad():
                out.mul_(2)
            if on:
                with pytest.raises(RuntimeError, match="modified by an inplace operation"):
                    torch.autograd.grad([out, denom], xs, [g_out, g_den])
            else:
                torch.autograd.grad([out, denom], xs, [g_out, g_den])
    finally:
        ua.set_save_output(True)
