"""What a stack's native passes must not change: every call that the module-by-module and operator-by-operator
passes take (replaced modules, hooks, autocast, float32 norms, odd masks) gives their result, and is refused
where they refuse it."""
import pytest
import torch
from torch import nn

from tests.test_gpu_t5_stack import _model as _fixture_model

pytestmark = pytest.mark.gpu


def _model(dtype=torch.bfloat16, **over):
    """A small model whose softmaxes are not one-hot (fan-in scaled weights)."""
    model = _fixture_model(dtype, **{**dict(d_model=128, num_heads=4, d_ff=256), **over})
    with torch.no_grad():
        for n, p in model.named_parameters():
            if p.dim() > 1 and "shared" not in n:
                p.mul_(12.5 * p.shape[-1] ** -0.5)
    return model


def _ids(B, L, seed=0):
    return torch.randint(0, 128, (B, L), generator=torch.Generator().manual_seed(seed)).cuda()


def _mask(lens, L):
    return (torch.arange(L)[None] < torch.tensor(lens)[:, None]).long().cuda()


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-6)).item()


def _by_modules(stack):
    """Context: the stack runs module by module (a hook on one of its modules selects that path)."""
    import contextlib

    @contextlib.contextmanager
    def cm():
        h = stack.block[0].layer[0].SelfAttention.q.register_forward_hook(lambda *a: None)
        try:
            yield
        finally:
            h.remove()
    return cm()


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("width", [92, 108, 50, 200])
def test_a_mask_of_another_shape_than_the_rows_is_refused(width, grad):
    model = _model()
    ids, dec = _ids(2, 100), _ids(2, 20, 1)
    bad = _mask([width, width // 2], width)
    with torch.set_grad_enabled(grad):
        memory = model.encoder(ids)
        for call in (lambda: model.encoder(ids, attention_mask=bad),
                     lambda: model.decoder(dec, encoder_hidden_states=memory, encoder_attention_mask=bad),
                     lambda: model(ids, dec, attention_mask=bad),
                     lambda: model.encoder(ids, attention_mask=_mask([100, 90, 80], 100))):
            with pytest.raises((RuntimeError, ValueError, IndexError)):
                call()
    with torch.no_grad(), pytest.raises((RuntimeError, ValueError, IndexError)):
        model.encoder.forward_fused(ids, attention_mask=bad)
    torch.cuda.synchronize()


def test_a_memory_of_another_batch_than_the_rows_is_not_cut():
    model = _model()
    dec = _ids(2, 20, 1)
    with torch.no_grad():
        memory = model.encoder(_ids(4, 50))
        with pytest.raises((RuntimeError, ValueError)):
            model.decoder.forward_fused(dec, encoder_hidden_states=memory)
        # the modules view the memory's rows as the decoder's batch; whatever they give, the stack gives too
        got = model.decoder(dec, encoder_hidden_states=memory)
        with _by_modules(model.decoder):
            want = model.decoder(dec, encoder_hidden_states=memory)
    assert _rel(got, want) < 2e-2


@torch.no_grad()
def test_given_operators_serve_masked_and_packed_passes_too():
    from turbot5_b200.t5 import _FusedOps

    class Counting(_FusedOps):
        calls = 0

        @staticmethod
        def rms_layer_norm(*a):
            Counting.calls += 1
            return _FusedOps.rms_layer_norm(*a)

    model = _model()
    ids, dec = _ids(3, 70), _ids(3, 9, 1)
    mask = _mask([70, 31, 1], 70)
    want = model.encoder.forward_fused(ids, attention_mask=mask)
    got = model.encoder.forward_fused(ids, attention_mask=mask, ops=Counting)
    assert Counting.calls == 1 and _rel(got, want) < 1e-2 and torch.count_nonzero(got[1, 31:]) == 0
    packed, plan = model.encoder.forward_fused(ids, attention_mask=mask, packed_rows=110, return_packed=True, ops=Counting)
    states = model.encoder.forward_fused(ids, attention_mask=mask, packed_rows=110, return_packed=True)[0]
    want = model.decoder.forward_fused(dec, encoder_hidden_states=states, encoder_plan=plan)
    got = model.decoder.forward_fused(dec, encoder_hidden_states=packed, encoder_plan=plan, ops=Counting)
    assert _rel(got, want) < 1e-2


def test_inference_under_autocast():
    model = _model()
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    mask = _mask([70, 31], 70)
    with torch.no_grad():
        want, want_masked = model(ids, dec), model(ids, dec, attention_mask=mask)
        with torch.autocast("cuda", torch.bfloat16):
            assert _rel(model(ids, dec), want) < 2e-2
            assert _rel(model(ids, dec, attention_mask=mask), want_masked) < 2e-2
            assert _rel(model.encoder.forward_fused(ids, attention_mask=mask, packed_rows=110),
                        model.encoder(ids, attention_mask=mask) * mask[..., None]) < 2e-2
            tokens = model.generate(ids, attention_mask=mask, max_new_tokens=4, use_cuda_graph=False)
    assert tokens.shape == (2, 4)


@torch.no_grad()
@pytest.mark.parametrize("what", ["norms", "table", "strided"])
def test_inference_with_weights_the_native_pass_does_not_take(what):
    """Norm weights or a bias table in float32 beside 16-bit matrices, and weights that are not contiguous: no
    farther from the float32 model than the native pass is (rounded at the same points or at fewer; half as
    much again for the chance of single roundings, which these softmaxes magnify)."""
    model = _model()
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    mask = _mask([70, 31], 70)
    exact = _model(torch.float32)
    for p, e in zip(model.parameters(), exact.parameters()):
        e.copy_(p)
    exact, exact_masked = exact(ids, dec), exact(ids, dec, attention_mask=mask)
    bound, bound_masked = 1.5 * _rel(model(ids, dec), exact), 1.5 * _rel(model(ids, dec, attention_mask=mask), exact_masked)
    for n, p in model.named_parameters():
        if (what == "norms" and "layer_norm" in n) or (what == "table" and "relative_attention_bias" in n):
            p.data = p.data.float()
        if what == "strided" and p.dim() == 2 and ("SelfAttention" in n or "DenseReluDense" in n) and "relative" not in n:
            p.data = p.data.t().contiguous().t()
    assert _rel(model(ids, dec), exact) <= bound < 0.2
    assert _rel(model(ids, dec, attention_mask=mask), exact_masked) <= bound_masked < 0.2


class _Squared(nn.Module):
    """A feed-forward layer with the names of the plain one and another activation."""

    def __init__(self, old):
        super().__init__()
        self.wi, self.wo = old.wi, old.wo

    def forward(self, x):
        return self.wo(torch.relu(self.wi(x)).square())


def test_a_replaced_feed_forward_module_is_the_one_that_runs():
    model = _model(feed_forward_proj="relu")
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    plain = model.encoder.forward_fused(ids)
    for stack in (model.encoder, model.decoder):
        for blk in stack.block:
            blk.layer[-1].DenseReluDense = _Squared(blk.layer[-1].DenseReluDense)
    with torch.no_grad():
        got, want = model.encoder.forward_fused(ids), model.encoder(ids)
        assert _rel(got, want) < 2e-2 and _rel(plain, want) > 5e-2
        logits = model(ids, dec)
        want = model.logits(model.decoder(dec, encoder_hidden_states=want))
        assert _rel(logits, want) < 3e-2
        masked = model(ids, dec, attention_mask=_mask([70, 70], 70))
        assert _rel(masked, want) < 3e-2


def test_hooks_and_biases_of_a_feed_forward_layer_are_honoured():
    model = _model(feed_forward_proj="relu")
    ids = _ids(2, 70)
    want_plain = model.encoder.forward_fused(ids)
    seen = []
    handle = model.encoder.block[0].layer[-1].DenseReluDense.register_forward_hook(lambda *a: seen.append(1))
    got = model.encoder.forward_fused(ids)
    handle.remove()
    assert seen and _rel(got, want_plain) < 2e-2
    wi = model.encoder.block[1].layer[-1].DenseReluDense.wi
    wi.bias = nn.Parameter(torch.full((256,), 0.5, device="cuda", dtype=torch.bfloat16))
    with torch.no_grad():
        want = model.encoder(ids)
    assert _rel(model.encoder.forward_fused(ids), want) < 2e-2 < _rel(want_plain, want)


def _shift_weights(model, factor=0.5, data=False):
    for stack in (model.encoder, model.decoder):
        for blk in stack.block:
            sa = blk.layer[0].SelfAttention
            for p in (sa.q.weight, sa.v.weight, blk.layer[-1].DenseReluDense.wi_0.weight):
                p.data.mul_(factor) if data else p.mul_(factor)


def test_weights_made_under_inference_mode_are_never_stale():
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    with torch.inference_mode():
        model = _model()
        model(ids, dec)
        _shift_weights(model)
        got, states = model(ids, dec), model.encoder(ids)
        tokens, last = model.greedy_decode(states, 7)
        fresh = _model()
        _shift_weights(fresh)
        assert torch.equal(got, fresh(ids, dec)) and torch.equal(states, fresh.encoder(ids))
        want_tokens, want_last = fresh.greedy_decode(states, 7)
        assert torch.equal(tokens, want_tokens) and torch.equal(last, want_last)


@torch.no_grad()
def test_a_pass_of_the_module_interface_sees_updates_that_no_version_counter_shows():
    """`p.data` updates (optimisers, moving averages, collectives) leave a parameter's version as it is; passes
    that ran module by module saw them."""
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    model, fresh = _model(), _model()
    states = model.encoder(ids)
    model.decoder(dec, encoder_hidden_states=states)
    model.greedy_decode(states, 7)
    _shift_weights(model, data=True)
    _shift_weights(fresh)
    got, want = model.encoder(ids), fresh.encoder(ids)
    assert torch.equal(got, want)
    assert torch.equal(model.decoder(dec, encoder_hidden_states=got), fresh.decoder(dec, encoder_hidden_states=want))
    for a, b in zip(model.greedy_decode(got, 7), fresh.greedy_decode(want, 7)):
        assert torch.equal(a, b)


@torch.no_grad()
def test_a_first_pass_inside_a_capture_leaves_nothing_behind_for_later_passes():
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    want = _model()(ids, dec)                  # library handles exist from here on
    model = _model()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = model(ids, dec)
    assert torch.equal(model(ids, dec), want)  # before any replay: nothing that the graph would write may be read
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    # updated weights: eager passes and replays both see them, and a replay reads no memory that was given back
    _shift_weights(model)
    fresh = _model()
    _shift_weights(fresh)
    want = fresh(ids, dec)
    assert torch.equal(model(ids, dec), want)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@torch.no_grad()
def test_passes_on_several_streams_share_the_stacked_weights_in_order():
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    model = _model()
    want = _model()(ids, dec)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    filler = torch.randn(8192, 8192, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        for _ in range(4):
            filler @ filler                    # the stacked copies are built behind some milliseconds of work
        first = model(ids, dec)
    with torch.cuda.stream(b):
        second = model(ids, dec)
    torch.cuda.synchronize()
    assert torch.equal(first, want) and torch.equal(second, want)


def _into_flat_buffer(model, offset):
    """Every parameter a view into one buffer, each starting `offset` elements past a 16-byte boundary."""
    params = list(model.parameters())
    room = [(p.numel() + 15) // 8 * 8 + 8 for p in params]
    flat = torch.zeros(sum(room) + 8, device="cuda", dtype=params[0].dtype)
    at = 0
    for p, n in zip(params, room):
        view = flat[at + offset:at + offset + p.numel()].view_as(p)
        view.copy_(p.data)
        p.data = view
        at += n
    return model


@pytest.mark.parametrize("offset", [1, 4])
def test_parameters_that_are_views_at_odd_offsets(offset):
    """Sharding and data-parallel wrappers keep parameters in flat buffers; 16-byte loads and bulk copies must not
    meet them there.  (The library takes other products for such weights: sums in another order, so no farther
    from the float32 model than the aligned run, and half as much again for the chance of single roundings.)"""
    ids, dec, mask = _ids(3, 70), _ids(3, 9, 1), _mask([70, 31, 2], 70)
    aligned, model = _model(), _into_flat_buffer(_model(), offset)
    exact = _model(torch.float32)
    with torch.no_grad():
        for p, e in zip(aligned.parameters(), exact.parameters()):
            e.copy_(p)
        exact = exact(ids, dec, attention_mask=mask)
        assert _rel(model(ids, dec, attention_mask=mask), exact) <= 1.5 * _rel(aligned(ids, dec, attention_mask=mask), exact) < 0.2
        states = aligned.encoder(ids)
        for graph in (False, True):
            tokens, last = model.greedy_decode(states, 8, use_cuda_graph=graph)
            dec_in = torch.cat([torch.zeros((3, 1), dtype=torch.long, device="cuda"), tokens[:, :-1]], dim=1)
            full = aligned.logits(aligned.decoder(dec_in, encoder_hidden_states=states))
            assert _rel(last[:, -1], full[:, -1]) < 4e-2
    embedded = aligned.shared(ids).detach()
    room = torch.zeros(embedded.numel() + 8, device="cuda", dtype=embedded.dtype)
    odd = room[offset:offset + embedded.numel()].view_as(embedded).copy_(embedded)
    grads = []
    for m, x in ((aligned, embedded), (model, odd)):
        out = m.encoder(inputs_embeds=x.requires_grad_())
        dout = torch.randn(out.shape, generator=torch.Generator().manual_seed(5)).to(out)
        grads.append(torch.autograd.grad(out, [x] + list(m.encoder.block.parameters()), dout))
    for a, b in zip(*grads):
        assert _rel(b, a) < 4e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("offset", [0, 1, 4])
@pytest.mark.parametrize("d", [512, 768, 1024, 500])
def test_norm_backward_with_a_residual_gradient_at_any_offset(offset, d, dtype):
    from turbot5_b200 import _native as nat
    rows, eps = 37, 1e-6
    g = torch.Generator().manual_seed(7)
    x, dy, add = (torch.randn((rows, d), generator=g).to("cuda", dtype) for _ in range(3))
    w = (1 + 0.1 * torch.randn(d, generator=g)).to("cuda", dtype)
    room = torch.zeros(rows * d + 8, device="cuda", dtype=dtype)
    odd = room[offset:offset + rows * d].view(rows, d).copy_(add)
    dx, dw = torch.empty_like(x), torch.zeros(d, device="cuda")
    code = nat.dtype_code(dtype)
    st = nat.lib().t5b_rmsnorm_bwd_add(x.data_ptr(), w.data_ptr(), dy.data_ptr(), odd.data_ptr(), dx.data_ptr(), dw.data_ptr(),
                                       rows, d, d, d, d, code, code, eps, nat.stream_ptr(x.device))
    assert st == 0
    xf, wf = x.double().requires_grad_(), w.double().requires_grad_()
    (xf * torch.rsqrt(xf.square().mean(-1, keepdim=True) + eps) * wf).backward(dy.double())
    want = xf.grad + add.double()
    # one rounding of the result (2^-9 or 2^-12 relative), float32 sums before it
    assert (dx.double() - want).abs().max().item() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * want.abs().max().item()
    # the kernel rounds x * rstd as the forward pass does: that error is at most one half ulp a term
    assert _rel(dw, wf.grad) < 2.0 ** -8


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("width", [64, 512])
def test_layers_of_different_widths(width, grad):
    """One layer's feed-forward pruned or widened (plain modules of other sizes): run module by module."""
    model = _model()
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    g = torch.Generator().manual_seed(3)
    for stack in (model.encoder, model.decoder):
        ff = stack.block[1].layer[-1].DenseReluDense
        for name, shape in (("wi_0", (width, 128)), ("wi_1", (width, 128)), ("wo", (128, width))):
            linear = nn.Linear(shape[1], shape[0], bias=False)
            linear.weight.data = torch.randn(shape, generator=g) * shape[1] ** -0.5
            setattr(ff, name, linear.cuda().bfloat16())
    with torch.set_grad_enabled(grad):
        states = model.encoder(ids)
        hidden = model.decoder(dec, encoder_hidden_states=states)
        with _by_modules(model.encoder), _by_modules(model.decoder):
            want_states = model.encoder(ids)
            want = model.decoder(dec, encoder_hidden_states=want_states)
    assert torch.equal(states, want_states) and torch.equal(hidden, want)
    with torch.no_grad():
        fused = model.decoder.forward_fused(dec, encoder_hidden_states=model.encoder.forward_fused(ids))
        assert _rel(fused, want) < 4e-2
        tokens, last = model.greedy_decode(states.detach(), 5)
        with _by_modules(model.decoder):
            want_tokens, want_last = model.greedy_decode(states.detach(), 5)
    assert torch.equal(tokens, want_tokens) and torch.equal(last, want_last)


class _Held(torch.Tensor):
    """A weight that lives in another tensor, as quantised and sharded weights do."""

    @staticmethod
    def __new__(cls, inner):
        return torch.Tensor._make_wrapper_subclass(cls, inner.shape, dtype=inner.dtype, device=inner.device,
                                                   strides=inner.stride())

    def __init__(self, inner):
        self.inner = inner

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        from torch.utils._pytree import tree_map_only
        plain = tree_map_only(_Held, lambda t: t.inner, (args, kwargs or {}))
        out = func(*plain[0], **plain[1])
        return _Held(out) if func is torch.ops.aten.detach.default else out


@torch.no_grad()
def test_weights_that_are_tensor_subclasses():
    model = _model()
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    want = model.decoder(dec, encoder_hidden_states=model.encoder(ids))
    for stack in (model.encoder, model.decoder):
        q = stack.block[0].layer[0].SelfAttention.q
        q.weight = nn.Parameter(_Held(q.weight.detach()), requires_grad=False)
    got = model.decoder(dec, encoder_hidden_states=model.encoder(ids))
    assert _rel(got, want) < 4e-2


@torch.no_grad()
@pytest.mark.parametrize("B,over,dtype", [
    (2, dict(d_model=2048, num_heads=32, d_ff=5120), torch.float16),        # a normed product of several tiles
    (64, dict(d_model=2048, num_heads=4), torch.bfloat16),                  # 64 rows beside a wide LM head
    (33, dict(d_model=1664, num_heads=4), torch.float16),
    (2, dict(d_ff=8192), torch.bfloat16), (3, dict(d_ff=6624, feed_forward_proj="relu"), torch.float16),
    (1, dict(d_model=2016, num_heads=2), torch.bfloat16), (17, dict(d_model=1728, num_heads=2), torch.bfloat16),
    (40, dict(d_model=1696, num_heads=2), torch.float16)])
def test_wide_decoders_generate(B, over, dtype):
    """Widths whose largest tiles do not fit in shared memory: smaller tiles serve them.  No row of the last logits
    is farther from the float32 model over the same tokens than the worst row of the uncached 16-bit pass (half as
    much again for the chance of single roundings), and a chosen token trails the best by no more than two such elements' errors."""
    model = _model(dtype, num_layers=1, num_decoder_layers=1, **over)
    exact = _model(torch.float32, num_layers=1, num_decoder_layers=1, **over)
    for p, e in zip(model.parameters(), exact.parameters()):
        e.copy_(p)
    g = torch.Generator().manual_seed(31)
    enc = torch.randn((B, 40, model.cfg.d_model), generator=g).to("cuda", dtype)
    tokens, last = model.greedy_decode(enc, 7, use_cuda_graph=True)
    dec_in = torch.cat([torch.zeros((B, 1), dtype=torch.long, device="cuda"), tokens[:, :-1]], dim=1)
    full = model.logits(model.decoder(dec_in, encoder_hidden_states=enc)).float()
    exact = exact.logits(exact.decoder(dec_in, encoder_hidden_states=enc.float()))
    rows = lambda a, b: ((a.float() - b).norm(dim=-1) / b.norm(dim=-1)).max().item()
    assert rows(last[:, -1], exact[:, -1]) <= 1.5 * rows(full, exact) < 0.2
    chosen = exact.gather(-1, tokens[..., None])[..., 0]
    assert (exact.max(-1).values - chosen).max().item() <= 4 * (full - exact).abs().max().item()


class _Adapter(nn.Module):
    """Another feed-forward layer altogether: no child of the plain one's names."""

    def __init__(self, d):
        super().__init__()
        self.scale = nn.Parameter(torch.full((d,), 0.25, device="cuda", dtype=torch.bfloat16))

    def forward(self, x):
        return x * self.scale


class _NoWeight(nn.Module):
    def __init__(self, linear):
        super().__init__()
        self.inner = linear

    def forward(self, x):
        return self.inner(x)


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("what", ["feed-forward", "projection", "norm", "instance forward", "eps"])
def test_replaced_modules_run_as_modules(what, grad):
    """A module of another class, without the children or the weight that the plain one has, with a `forward`
    of its own in the instance, or with another epsilon: run by calling it, as before."""
    model = _model()
    ids, dec = _ids(2, 70), _ids(2, 9, 1)
    calls = []

    class Norm(nn.Module):
        def __init__(self, d):
            super().__init__()
            self.g = nn.Parameter(torch.ones(d, device="cuda", dtype=torch.bfloat16))

        def forward(self, x):
            calls.append(1)
            return x * self.g

    for stack in (model.encoder, model.decoder):
        blk = stack.block[1]
        if what == "feed-forward":
            blk.layer[-1].DenseReluDense = _Adapter(128)
        elif what == "projection":
            blk.layer[0].SelfAttention.k = _NoWeight(blk.layer[0].SelfAttention.k)
        elif what == "norm":
            blk.layer[-1].layer_norm = Norm(128)
        elif what == "eps":
            blk.layer[-1].layer_norm.eps = 10.0
        else:
            blk.layer[-1].DenseReluDense.forward = lambda x: x * 0.25
    with torch.set_grad_enabled(grad):
        states = model.encoder(ids)
        hidden = model.decoder(dec, encoder_hidden_states=states)
        if what == "norm":
            assert len(calls) == 2
        with _by_modules(model.encoder), _by_modules(model.decoder):
            want_states = model.encoder(ids)
            want = model.decoder(dec, encoder_hidden_states=want_states)
        assert torch.equal(states, want_states) and torch.equal(hidden, want)
    with torch.no_grad():
        # (the cached steps by operators read the projections' weights themselves: they never took such a module)
        if what != "projection":
            tokens, last = model.greedy_decode(states.detach(), 5)
            with _by_modules(model.decoder):
                want_tokens, want_last = model.greedy_decode(states.detach(), 5)
            assert torch.equal(tokens, want_tokens) and torch.equal(last, want_last)


def test_a_wrapped_encoder_is_called_in_training():
    class Wrapped(nn.Module):
        def __init__(self, inner):
            super().__init__()
            self.inner, self.calls = inner, 0

        def forward(self, *a, **k):
            self.calls += 1
            return self.inner(*a, **k)

        def __getattr__(self, name):
            try:
                return super().__getattr__(name)
            except AttributeError:
                return getattr(super().__getattr__("inner"), name)

    model = _model()
    ids, dec, mask = _ids(2, 70), _ids(2, 9, 1), _mask([70, 31], 70)
    want = model(ids, dec, attention_mask=mask)
    model.encoder = Wrapped(model.encoder)
    got = model(ids, dec, attention_mask=mask)
    assert model.encoder.calls == 1 and _rel(got, want) < 2e-2


def test_a_masked_training_step_can_be_captured():
    """No pass reads a count back where that is forbidden: in a capture, and under the synchronisation check."""
    model = _model().train()
    ids, dec, mask = _ids(3, 70), _ids(3, 9, 1), _mask([70, 31, 2], 70)
    params = list(model.parameters())

    def step():
        logits = model(ids, dec, attention_mask=mask)
        return torch.autograd.grad(logits.float().square().mean(), params)
    want = step()
    torch.cuda.set_sync_debug_mode("error")
    try:
        step()
    finally:
        torch.cuda.set_sync_debug_mode("default")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert _rel(a, b) < 4e-2


def test_saved_tensor_hooks_see_the_activations_of_a_stack():
    """Offloading and checkpointing work by hooks on what autograd saves: under them a stack runs module by module,
    so every activation goes through the hooks."""
    model = _model().train()
    ids, dec, mask = _ids(3, 70), _ids(3, 9, 1), _mask([70, 31, 2], 70)
    params = list(model.parameters())
    own = {p.untyped_storage().data_ptr() for p in params}

    def grads():
        logits = model(ids, dec, attention_mask=mask)
        return torch.autograd.grad(logits.float().square().mean(), params)
    want = grads()
    packed = []

    def pack(t):
        if t.untyped_storage().data_ptr() not in own:
            packed.append(tuple(t.shape))
        return t
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        got = grads()
    rows = [s for s in packed if len(s) >= 2 and s[-1] == 256]    # feed-forward rows: two products a layer at least
    assert len(rows) >= 2 * 4, packed
    for a, b in zip(got, want):
        assert _rel(a, b) < 4e-2
    with torch.autograd.graph.save_on_cpu(pin_memory=True):
        got = grads()
    for a, b in zip(got, want):
        assert _rel(a, b) < 4e-2
    from torch.utils.checkpoint import checkpoint
    embedded = model.encoder.embed_tokens(ids).detach().requires_grad_()
    out = model.encoder(inputs_embeds=embedded)
    dout = torch.randn(out.shape, generator=torch.Generator().manual_seed(5)).to(out)
    want = torch.autograd.grad(out, embedded, dout)[0]
    out = checkpoint(lambda e: model.encoder(inputs_embeds=e), embedded, use_reentrant=False)
    assert _rel(torch.autograd.grad(out, embedded, dout)[0], want) < 4e-2


def test_forward_mode_inputs_that_ask_for_gradients_are_refused():
    import torch.autograd.forward_ad as fw
    import turbot5_b200 as t5b
    model = _model()
    q = torch.randn(1, 2, 64, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.ones(128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    x = torch.randn(2, 16, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    plan = t5b.get_unpad_plan(_mask([16, 3], 16))
    with fw.dual_level():
        dual = lambda t: fw.make_dual(t, torch.ones_like(t))
        for call in (lambda: t5b.flash_attention_with_fusing_bias(dual(q), q, q, None),
                     lambda: t5b.rms_layer_norm(dual(x), w),
                     lambda: t5b.unpad_rows(dual(x), plan),
                     lambda: model.encoder(inputs_embeds=dual(x))):
            with pytest.raises((RuntimeError, NotImplementedError)):
                call()


def _same_until_a_near_tie(model, states, tokens, other):
    """Two greedy runs of the same model: equal tokens, or the first difference of a row is at a step where the two
    tokens' logits in an uncached pass over the common prefix are within what 16-bit passes differ by."""
    for b in range(tokens.shape[0]):
        diff = (tokens[b] != other[b]).nonzero()
        if diff.numel() == 0:
            continue
        t = int(diff[0])
        dec_in = torch.cat([torch.zeros((1, 1), dtype=torch.long, device="cuda"), tokens[b:b + 1, :t]], dim=1)
        logits = model.logits(model.decoder(dec_in, encoder_hidden_states=states[b:b + 1]))[0, -1].float()
        gap = (logits[tokens[b, t]] - logits[other[b, t]]).abs().item()
        assert gap <= 0.1 * logits.abs().mean().item(), (b, t, gap)


@torch.no_grad()
@pytest.mark.parametrize("ff", ["gated-gelu", "relu"])
@pytest.mark.parametrize("B,steps,why", [(3, 7, "hook"), (65, 7, "rows"), (1, 530, "hook")])
def test_the_decoding_paths_without_the_step_kernels(B, steps, why, ff):
    """What serves models and batches that the step kernels do not take: the eager cached steps and the captured
    static step, against each other and against the step kernels where those run (530 cached keys: the captured
    self attention splits them)."""
    from turbot5_b200 import _native as nat
    from turbot5_b200.t5 import _native_decoding
    model = _model(feed_forward_proj=ff)
    states = model.encoder(_ids(B, 120, 6))
    native = None
    if why == "hook":
        native, _ = model.greedy_decode(states, steps)
        handle = model.decoder.block[0].layer[0].SelfAttention.q.register_forward_hook(lambda *a: None)
    assert _native_decoding(model, states, steps) is None
    eager, eager_last = model.greedy_decode(states, steps)
    graphed, graphed_last = model.greedy_decode(states, steps, use_cuda_graph=True)
    if steps > 500:
        assert nat.lib().t5b_decode_num_splits(B, 4, steps) > 1
    if why == "hook":
        handle.remove()
        _same_until_a_near_tie(model, states, native, eager)
    _same_until_a_near_tie(model, states, graphed, eager)
    same = (eager == graphed).all(1)
    assert same.float().mean() >= 0.5 or steps > 500
    if same.any():
        assert _rel(graphed_last[same], eager_last[same]) < 6e-2


@torch.no_grad()
def test_float32_decoding_through_a_graph():
    model = _model(torch.float32)
    states = model.encoder(_ids(2, 60))
    eager, eager_last = model.greedy_decode(states, 9)
    graphed, graphed_last = model.greedy_decode(states, 9, use_cuda_graph=True)
    assert torch.equal(eager, graphed) and _rel(graphed_last, eager_last) < 1e-4
