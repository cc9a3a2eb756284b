"""The thin T5 stack (CUDA kernels + cuBLAS linears) against the reference's whole-model fixture
and against the stack oracle."""
import pytest
import torch

from oracle import t5_oracle as orc
from tests.helpers import TINY_T5, load, seed_named_parameters, tiny_t5_inputs

pytestmark = pytest.mark.gpu


def _model(dtype, **over):
    from turbot5_b200.t5 import T5ForConditionalGeneration, T5StackConfig
    cfg = T5StackConfig(**{**TINY_T5, **over})
    model = seed_named_parameters(T5ForConditionalGeneration(cfg), 0)
    return model.cuda().to(dtype).eval()


def test_fp32_stack_matches_reference_model_fixture():
    z = load("stack.npz")
    model = _model(torch.float32)
    ids, dec = tiny_t5_inputs()
    with torch.no_grad():
        enc = model.encoder(ids.cuda())
        logits = model(ids.cuda(), dec.cuda())
        mask = torch.from_numpy(z["mask"]).cuda()
        enc_m = model.encoder(ids.cuda(), attention_mask=mask)
        logits_m = model(ids.cuda(), dec.cuda(), attention_mask=mask)
        tokens, last = model.greedy_decode(enc, 4)
    assert (enc.cpu() - torch.from_numpy(z["encoder"])).abs().max().item() < 2e-4
    assert (logits.cpu() - torch.from_numpy(z["logits"])).abs().max().item() < 2e-4
    valid = torch.from_numpy(z["mask"]).bool()
    assert (enc_m.cpu() - torch.from_numpy(z["encoder_masked"]))[valid].abs().max().item() < 2e-4
    assert (logits_m.cpu() - torch.from_numpy(z["logits_masked"])).abs().max().item() < 2e-4
    assert torch.equal(tokens.cpu(), torch.from_numpy(z["greedy_tokens"]))
    assert (last[:, -1].cpu() - torch.from_numpy(z["greedy_logits"][:, 3])).abs().max().item() < 2e-4


def test_bf16_stack_close_to_fp32_oracle():
    # wider model so the tensor-core kernels are the ones that run (bf16, d_kv 64)
    over = dict(d_model=128, num_heads=4, d_ff=256)
    model = _model(torch.bfloat16, **over)
    w = {k: v.detach().float().cpu() for k, v in model.state_dict().items()}
    cfg = {**TINY_T5, **over}
    g = torch.Generator().manual_seed(3)
    ids = torch.randint(0, 128, (2, 300), generator=g)
    dec = torch.randint(0, 128, (2, 150), generator=g)
    with torch.no_grad():
        enc = model.encoder(ids.cuda())
        logits = model(ids.cuda(), dec.cuda())
    enc_want, logits_want = orc.t5_model_logits(w, cfg, ids, dec)
    # every linear, norm and residual of 2 + 2 layers runs in bf16 here against an all-float32
    # oracle: compare in relative terms (the kernels themselves are held to the tight
    # tolerances in the other test files)
    rel = lambda a, b: ((a.float().cpu() - b).abs().mean() / b.abs().mean()).item()
    assert rel(enc, enc_want) < 2e-2
    assert rel(logits, logits_want) < 1e-1


def test_cached_greedy_equals_uncached_recompute_bf16():
    model = _model(torch.bfloat16, d_model=128, num_heads=4, d_ff=256)
    g = torch.Generator().manual_seed(4)
    ids = torch.randint(0, 128, (3, 200), generator=g).cuda()
    with torch.no_grad():
        enc = model.encoder(ids)
        tokens, last = model.greedy_decode(enc, 6)
        # teacher-forced full pass over the generated prefix gives the same last-step logits
        dec_in = torch.cat([torch.zeros((3, 1), dtype=torch.long, device="cuda"), tokens[:, :-1]], dim=1)
        full = model.logits(model.decoder(dec_in, encoder_hidden_states=enc))
    assert (full[:, -1].float() - last[:, -1].float()).abs().max().item() < 0.15
    assert (full[:, -1].argmax(-1) == tokens[:, -1]).float().mean().item() >= 0.66


def test_state_dict_names_follow_hf_layout():
    from turbot5_b200.t5 import T5ForConditionalGeneration, T5StackConfig
    z = load("stack.npz")
    model = T5ForConditionalGeneration(T5StackConfig(**TINY_T5))
    assert sorted(n for n, _ in model.named_parameters()) == [str(x) for x in z["param_names"]]


def test_cuda_graph_decoding_equals_eager_decoding():
    model = _model(torch.bfloat16, d_model=128, num_heads=4, d_ff=256)
    g = torch.Generator().manual_seed(5)
    ids = torch.randint(0, 128, (3, 300), generator=g).cuda()
    with torch.no_grad():
        enc = model.encoder(ids)
        eager_tokens, eager_last = model.greedy_decode(enc, 7)
        graph_tokens, graph_last = model.greedy_decode(enc, 7, use_cuda_graph=True)
    assert torch.equal(eager_tokens, graph_tokens)
    assert (eager_last.float() - graph_last.float()).abs().max().item() < 1e-2


def test_fused_encoder_packs_a_padded_batch_once():
    """forward_fused with the padding mask: the valid tokens are packed after the embedding, every layer runs
    on the packed rows, the result is scattered back -- same hidden states as the module path with the mask on
    the valid rows, zeros on the padded ones; with and without the caller's bound on the token count."""
    model = _model(torch.bfloat16, d_model=128, num_heads=4, d_ff=256)
    g = torch.Generator().manual_seed(11)
    B, L = 4, 300
    lens = [300, 171, 1, 64]
    ids = torch.randint(0, 128, (B, L), generator=g).cuda()
    mask = torch.zeros((B, L), dtype=torch.int64)
    for b, n in enumerate(lens):
        mask[b, :n] = 1
    mask = mask.cuda()
    with torch.no_grad():
        want = model.encoder(ids, attention_mask=mask)
        got = model.encoder.forward_fused(ids, attention_mask=mask)
        got2 = model.encoder.forward_fused(ids, attention_mask=mask, packed_rows=sum(lens) + 5)
    torch.cuda.synchronize()
    for b, n in enumerate(lens):
        assert (got[b, :n].float() - want[b, :n].float()).abs().max().item() < 6e-2, b
        assert (got[b, :n].float() - want[b, :n].float()).abs().mean().item() < 6e-3, b
        assert torch.count_nonzero(got[b, n:]) == 0
        assert torch.equal(got[b, :n], got2[b, :n])
    with torch.no_grad():          # a bound below the true count does not drop tokens silently
        bad = model.encoder.forward_fused(ids, attention_mask=mask, packed_rows=sum(lens) - 1)
    assert torch.isnan(bad[0, 0]).all()


def test_masked_inference_runs_packed_end_to_end():
    """A padded batch through the model in inference mode: the encoder packs the valid tokens once and the
    decoder's cross attention reads the packed states; same logits as the module path with the masks."""
    model = _model(torch.bfloat16, d_model=128, num_heads=4, d_ff=256)
    g = torch.Generator().manual_seed(12)
    B, L, Ld = 3, 260, 24
    lens = [260, 97, 5]
    ids = torch.randint(0, 128, (B, L), generator=g).cuda()
    dec = torch.randint(0, 128, (B, Ld), generator=g).cuda()
    mask = torch.zeros((B, L), dtype=torch.int64)
    for b, n in enumerate(lens):
        mask[b, :n] = 1
    mask = mask.cuda()
    with torch.no_grad():
        enc = model.encoder(ids, attention_mask=mask)
        want = model.logits(model.decoder(dec, encoder_hidden_states=enc, encoder_attention_mask=mask))
        got = model(ids, dec, attention_mask=mask)
    torch.cuda.synchronize()
    diff = (got.float() - want.float()).abs()
    assert diff.max().item() < 0.15 and diff.mean().item() < 1.5e-2, (diff.max().item(), diff.mean().item())


def test_generate_on_a_padded_batch_equals_the_step_by_step_module_path():
    """`generate`: packed encoder pass, cache, graph-captured steps -- the same tokens as the encoder module
    with the mask followed by eager cached decoding with the key lengths."""
    model = _model(torch.bfloat16, d_model=128, num_heads=4, d_ff=256)
    g = torch.Generator().manual_seed(13)
    B, L = 3, 200
    lens = [200, 61, 9]
    ids = torch.randint(0, 128, (B, L), generator=g).cuda()
    mask = torch.zeros((B, L), dtype=torch.int64)
    for b, n in enumerate(lens):
        mask[b, :n] = 1
    mask = mask.cuda()
    with torch.no_grad():
        enc = model.encoder(ids, attention_mask=mask)
        want, _ = model.greedy_decode(enc, 6, encoder_seqlens=torch.tensor(lens, dtype=torch.int32, device="cuda"))
    got = model.generate(ids, attention_mask=mask, max_new_tokens=6)
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_cuda_graph_forward_equals_eager_forward():
    """The whole teacher-forced pass as one graph: same logits as the eager pass, for two different
    inputs through the same graph (the ids are copied into the graph's buffers), wrong shapes refused."""
    from turbot5_b200.t5 import GraphedForward
    model = _model(torch.bfloat16, d_model=128, num_heads=4, d_ff=256)
    g = torch.Generator().manual_seed(8)
    graphed = GraphedForward(model, 3, 260, 24)
    for _ in range(2):
        ids = torch.randint(0, 128, (3, 260), generator=g).cuda()
        dec = torch.randint(0, 128, (3, 24), generator=g).cuda()
        with torch.no_grad():
            want = model(ids, dec)
        got = graphed(ids, dec)
        torch.cuda.synchronize()
        assert (got.float() - want.float()).abs().max().item() < 1e-2
    with pytest.raises(ValueError):
        graphed(ids[:2], dec[:2])
    got = model.forward_cuda_graph(ids, dec)          # the per-shape cache on the model
    again = model.forward_cuda_graph(ids, dec)
    torch.cuda.synchronize()
    assert got is again and (got.float() - want.float()).abs().max().item() < 1e-2


def test_cuda_graph_decoding_with_a_long_cache_splits_the_keys():
    """A cache long enough that the captured self-attention launch splits the keys (the split count
    comes from the capacity and stays the same in every replay): tokens as in eager decoding."""
    from turbot5_b200 import _native as nat
    model = _model(torch.bfloat16, d_model=128, num_heads=4, d_ff=256)
    steps = 530
    assert nat.lib().t5b_decode_num_splits(1, 4, steps) > 1
    ids = torch.randint(0, 128, (1, 200), generator=torch.Generator().manual_seed(6)).cuda()
    with torch.no_grad():
        enc = model.encoder(ids)
        eager_tokens, eager_last = model.greedy_decode(enc, steps)
        graph_tokens, graph_last = model.greedy_decode(enc, steps, use_cuda_graph=True)
    # bf16 logits of near-ties may order differently between the two launch sequences; once a token
    # differs the continuations diverge, so compare up to the first difference and require it late
    same = (eager_tokens == graph_tokens)[0]
    first_diff = int((~same).float().argmax()) if not bool(same.all()) else steps
    assert first_diff >= 64, first_diff
    if first_diff == steps:
        assert (eager_last.float() - graph_last.float()).abs().max().item() < 5e-2


def test_training_step_through_the_stack_gives_finite_gradients_everywhere():
    # encoder-decoder forward with a padding mask, cross-entropy loss, backward: every parameter
    # gets a finite, non-zero gradient through the CUDA attention, RMSNorm and unpad/pad kernels
    model = _model(torch.bfloat16, d_model=128, num_heads=2, d_ff=256).train()
    g = torch.Generator().manual_seed(9)
    ids = torch.randint(0, 128, (2, 150), generator=g).cuda()
    dec = torch.randint(0, 128, (2, 40), generator=g).cuda()
    mask = torch.ones((2, 150), dtype=torch.int64)
    mask[1, 90:] = 0
    enc = model.encoder(ids, attention_mask=mask.cuda())
    hid = model.decoder(dec, encoder_hidden_states=enc, encoder_attention_mask=mask.cuda())
    logits = model.logits(hid)
    loss = torch.nn.functional.cross_entropy(logits.float().view(-1, logits.shape[-1]), dec.view(-1))
    loss.backward()
    torch.cuda.synchronize()
    for name, prm in model.named_parameters():
        assert prm.grad is not None, name
        assert torch.isfinite(prm.grad.float()).all(), name
        assert prm.grad.float().abs().sum().item() > 0, name


def test_local_encoder_matches_the_full_encoder_when_one_block_covers_everything_but_the_padding_blocks():
    # a "local" encoder whose window is longer than the sequence differs from the full encoder only
    # by the reference's unmasked zero padding blocks; with blocks shorter than the sequence it must
    # differ; both run end to end and give finite outputs
    ids = torch.randint(0, 128, (2, 300), generator=torch.Generator().manual_seed(3)).cuda()
    full = _model(torch.bfloat16, d_model=128, num_heads=2, d_ff=256)
    local = _model(torch.bfloat16, d_model=128, num_heads=2, d_ff=256, attention_type="local", sliding_window=128)
    with torch.no_grad():
        a = full.encoder(ids)
        b = local.encoder(ids)
    assert a.shape == b.shape and torch.isfinite(b.float()).all()
    assert (a.float() - b.float()).abs().max().item() > 1e-3


@pytest.mark.parametrize("ff,masked,dtype", [("gated-gelu", False, torch.bfloat16), ("gated-gelu", True, torch.bfloat16),
                                             ("relu", True, torch.float16)])
def test_native_training_pass_gradients_equal_the_module_path(ff, masked, dtype):
    """The whole stack as one autograd node (packed when the batch is padded) against the same weights run
    module by module (a hook on one module selects that path).  Both round every activation and gradient to
    the 16-bit type at the same points up to the order of sums: a few 2^-8 (bf16) of each tensor's norm.
    The fixture's unit-variance weights make every softmax one-hot, and there a bf16 run's gradients differ
    from the float32 run's by more than their norm whichever path computes them; at 0.3 of them both paths
    are within 1.2 % of float32, and a sum or difference of two such runs within 4 %."""
    model = _model(dtype, d_model=256, num_heads=4, d_ff=192, feed_forward_proj=ff).train()
    with torch.no_grad():
        for n, p in model.named_parameters():
            if p.dim() > 1 and "shared" not in n:
                p.mul_(0.3)
    g = torch.Generator().manual_seed(21)
    B, L, Ld = 3, 150, 37
    ids, dec = torch.randint(0, 128, (B, L), generator=g).cuda(), torch.randint(0, 128, (B, Ld), generator=g).cuda()
    mask = None
    if masked:
        lens = torch.tensor([150, 61, 1])
        mask = (torch.arange(L)[None] < lens[:, None]).long().cuda()
    dout = torch.randn((B, Ld, 128), generator=g).to("cuda", dtype)

    def grads():
        model.zero_grad(set_to_none=True)
        logits = model(ids, dec, attention_mask=mask)
        logits.backward(dout)
        return logits.detach(), {n: p.grad.float() for n, p in model.named_parameters()}
    got_out, got = grads()
    handle = model.encoder.block[0].layer[0].SelfAttention.q.register_forward_hook(lambda *a: None)
    handle2 = model.decoder.block[0].layer[0].SelfAttention.q.register_forward_hook(lambda *a: None)
    want_out, want = grads()
    handle.remove(); handle2.remove()
    rel = lambda a, b: ((a - b).norm() / b.norm().clamp_min(1e-6)).item()
    assert rel(got_out.float(), want_out.float()) < 2e-2
    for n in want:
        assert rel(got[n], want[n]) < 4e-2, (n, rel(got[n], want[n]))


@pytest.mark.parametrize("B,L,steps,over,dtype", [
    (1, 7, 3, dict(), torch.bfloat16),                                             # one row, short memory: every split edge
    (3, 300, 20, dict(feed_forward_proj="relu"), torch.bfloat16),
    (17, 65, 5, dict(tie_word_embeddings=True), torch.bfloat16),                   # a second sixteen-row tile with one row
    (64, 129, 4, dict(), torch.float16),                                           # the largest batch
    (2, 200, 150, dict(d_model=1056, d_ff=2080, vocab_size=97), torch.bfloat16),   # rows over 1024, ragged vocabulary, split cache
    (5, 400, 6, dict(d_kv=128, num_heads=2), torch.bfloat16),
    (2, 90, 6, dict(d_kv=32, num_heads=3, d_ff=96), torch.bfloat16)])
def test_native_decoding_steps_equal_the_uncached_pass(B, L, steps, over, dtype):
    """Greedy decoding by the step kernels against the whole uncached decoder pass over the chosen tokens (other
    kernels throughout): same logits at the last step, and every chosen token is the best of its step or
    within the difference that two 16-bit passes show."""
    model = _model(dtype, **{**dict(d_model=128, num_heads=4, d_ff=256), **over})
    with torch.no_grad():
        for n, p in model.named_parameters():
            if p.dim() > 1 and "shared" not in n:
                p.mul_(p.shape[-1] ** -0.5)
    g = torch.Generator().manual_seed(31)
    enc = torch.randn((B, L, model.cfg.d_model), generator=g).to("cuda", dtype)
    lens = torch.randint(1, L + 1, (B,), generator=g, dtype=torch.int32)
    lens[0] = L
    mask = (torch.arange(L)[None] < lens[:, None]).long().cuda()
    from turbot5_b200.t5 import _native_decoding
    with torch.no_grad():
        assert _native_decoding(model, enc, steps, lens.cuda()) is not None
        tokens, last = model.greedy_decode(enc, steps, encoder_seqlens=lens.cuda(), use_cuda_graph=True)
        dec_in = torch.cat([torch.zeros((B, 1), dtype=torch.long, device="cuda"), tokens[:, :-1]], dim=1)
        full = model.logits(model.decoder(dec_in, encoder_hidden_states=enc, encoder_attention_mask=mask)).float()
    torch.cuda.synchronize()
    scale = full.abs().mean().item()
    assert (full[:, -1] - last[:, -1].float()).abs().max().item() < 0.08 * scale + 0.02
    chosen = full.gather(-1, tokens[..., None])[..., 0]
    assert (full.max(-1).values - chosen).max().item() < 0.08 * scale + 0.02


def test_graphed_decoding_replays_the_native_step():
    from turbot5_b200.t5 import GraphedDecoding
    model = _model(torch.bfloat16, d_model=128, num_heads=4, d_ff=256)
    enc = torch.randn((3, 200, 128), generator=torch.Generator().manual_seed(32)).cuda().bfloat16()
    want, last = model.greedy_decode(enc, 9)
    session = GraphedDecoding(model, enc, 9)
    for _ in range(2):
        session.rewind()
        for _ in range(9):
            session.step()
        torch.cuda.synchronize()
        assert torch.equal(session.tokens, want) and torch.equal(session.last_logits, last)
    with pytest.raises(RuntimeError):
        session.step()
