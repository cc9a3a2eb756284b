"""CPU-only checks of the C ABI library and the host-side logic (no kernel launches)."""
import ctypes
import os
import re

import numpy as np
import pytest
import torch

from tests.helpers import load

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol():
    from turbot5_b200 import _native as nat
    header = open(os.path.join(ROOT, "include", "turbot5_b200.h")).read()
    declared = set(re.findall(r"T5B_API[^;(]*?\b(t5b_\w+)\s*\(", header))
    assert declared == set(nat.SYMBOLS), declared ^ set(nat.SYMBOLS)
    L = ctypes.CDLL(nat.LIB_PATH)
    for name in declared:
        assert hasattr(L, name), name
    assert nat.lib().t5b_abi_version() == 1
    assert nat.lib().t5b_status_string(0) == b"ok"


def test_struct_layouts_match_header_field_order():
    from turbot5_b200 import _native as nat
    header = open(os.path.join(ROOT, "include", "turbot5_b200.h")).read()
    for cname, cls in (("t5b_attn_args", nat.AttnArgs), ("t5b_decode_args", nat.DecodeArgs),
                       ("t5b_attn_bwd_args", nat.AttnBwdArgs)):
        end = header.index("} " + cname + ";")
        body = header[header.rindex("typedef struct {", 0, end) + len("typedef struct {"):end]
        body = re.sub(r"/\*.*?\*/", "", body, flags=re.S)
        names = []
        for decl in body.split(";"):
            decl = decl.strip()
            if not decl:
                continue
            parts = decl.replace("*", " ").split(",")
            names.append(parts[0].split()[-1])
            names += [p.strip() for p in parts[1:]]
        assert names == [f[0] for f in cls._fields_], cname


def _header_fields(cname):
    header = open(os.path.join(ROOT, "include", "turbot5_b200.h")).read()
    end = header.index("} " + cname + ";")
    body = header[header.rindex("typedef struct {", 0, end) + len("typedef struct {"):end]
    body = re.sub(r"/\*.*?\*/", "", body, flags=re.S)
    fields = []
    for decl in body.split(";"):
        decl = decl.strip()
        if not decl:
            continue
        ctype = "ptr" if "*" in decl else decl.split()[0]
        parts = decl.replace("*", " ").split(",")
        fields.append((parts[0].split()[-1], ctype))
        fields += [(p.strip(), ctype) for p in parts[1:]]
    return fields


def test_integration_stub_struct_matches_header():
    """The ctypes struct a maintainer would paste from INTEGRATION.md has the header's fields, in
    order and with the header's types (a struct that is short or reordered corrupts calls)."""
    text = open(os.path.join(ROOT, "INTEGRATION.md")).read()
    start = text.index("class _AttnArgs(C.Structure)")
    end = text.index("_lib.t5b_attention_fwd.argtypes")
    scope = {"C": ctypes}
    exec(text[start:end], scope)
    stub = scope["_AttnArgs"]
    ctype_of = {"ptr": ctypes.c_void_p, "int64_t": ctypes.c_int64, "int32_t": ctypes.c_int32, "float": ctypes.c_float}
    want = [(n, ctype_of[t]) for n, t in _header_fields("t5b_attn_args")]
    assert [(n, t) for n, t in stub._fields_] == want
    from turbot5_b200 import _native as nat
    assert ctypes.sizeof(stub) == ctypes.sizeof(nat.AttnArgs)


def test_host_bucket_table_bit_exact_vs_reference_fixture():
    import turbot5_b200 as t5b
    z = load("buckets.npz")
    for nb, md, bidir, lo, hi in z["settings"]:
        key = f"nb{nb}_md{md}_{'bi' if bidir else 'uni'}"
        got = t5b.relative_position_bucket_table(int(nb), int(md), bool(bidir), int(lo), int(hi)).numpy()
        assert np.array_equal(got, z[key]), key


def test_host_bucket_table_rejects_bad_settings():
    import turbot5_b200 as t5b
    for nb, md in ((2, 128), (32, 0), (32, 4), (1024, 128)):
        with pytest.raises(RuntimeError):
            t5b.relative_position_bucket_table(nb, md, True)


def test_decode_split_heuristic_and_workspace_size():
    from turbot5_b200 import _native as nat
    L = nat.lib()
    assert L.t5b_decode_num_splits(64, 16, 8192) >= 2
    assert L.t5b_decode_num_splits(64, 16, 100) == 1
    assert L.t5b_decode_num_splits(1, 1, 1 << 20) == 64
    n = L.t5b_decode_workspace_bytes(64, 16, 1, 64, 8)
    assert n % 256 == 0 and n >= 64 * 16 * 8 * (64 + 2) * 4
    assert L.t5b_decode_workspace_bytes(0, 16, 1, 64, 8) == 0


def test_cpu_tensors_are_refused_not_silently_computed():
    import turbot5_b200 as t5b
    q = torch.zeros((1, 1, 4, 64))
    with pytest.raises(RuntimeError, match="CUDA"):
        t5b.flash_attention_with_fusing_bias(q, q, q, None)
    with pytest.raises(RuntimeError, match="CUDA"):
        t5b.rms_layer_norm(torch.zeros(2, 8), torch.ones(8))
    with pytest.raises(RuntimeError, match="CUDA"):
        t5b.get_unpad_plan(torch.ones((2, 3), dtype=torch.int64))


def test_entry_points_validate_arguments_without_a_device():
    from turbot5_b200 import _native as nat
    L = nat.lib()
    assert L.t5b_attention_fwd(None, None) == 5
    a = nat.AttnArgs()
    a.dtype, a.D, a.B, a.H, a.M, a.N = 7, 64, 1, 1, 1, 1
    assert L.t5b_attention_fwd(a, None) == 1           # dtype
    a.dtype, a.D = nat.BF16, 48
    assert L.t5b_attention_fwd(a, None) == 4           # head dim
    a.D, a.M = 64, -1
    assert L.t5b_attention_fwd(a, None) == 2           # shape
    a.M = 0
    assert L.t5b_attention_fwd(a, None) == 0           # empty problem: nothing to do
    a.M = 1
    assert L.t5b_attention_fwd(a, None) == 5           # null pointers
    assert L.t5b_rmsnorm_fwd(None, None, None, None, 1, 8, 8, 8, 0, 0, 1e-6, None) == 5
    assert L.t5b_decode_fwd(None, None) == 5
    assert L.t5b_unpad_plan(None, 1, 1, 1, None, None, None, None) == 5
    assert L.t5b_gather_rows(None, 16, None, 16, None, 1, 16, None) == 5


def test_registry_and_module_signature():
    import inspect
    import turbot5_b200 as t5b
    assert t5b.T5ATTENTION_TYPES["flash"] is t5b.T5FlashAttention
    sig = inspect.signature(t5b.T5FlashAttention.forward)
    assert list(sig.parameters)[1:] == ["hidden_states", "mask", "key_value_states", "position_bias",
                                        "past_key_value", "layer_head_mask", "query_length", "use_cache",
                                        "output_attentions"]
    sig = inspect.signature(t5b.flash_attention_with_fusing_bias)
    assert list(sig.parameters)[:8] == ["q", "k", "v", "bias", "causal", "sm_scale", "NUM_BUCKETS", "MAX_DISTANCE"]
    sig = inspect.signature(t5b.flash_attention_with_fusing_bias_varlen)
    assert list(sig.parameters)[:12] == ["q", "k", "v", "bias", "cu_seqlens_q", "cu_seqlens_k", "max_seqlen_q",
                                         "max_seqlen_k", "causal", "sm_scale", "NUM_BUCKETS", "MAX_DISTANCE"]


def test_host_bucket_table_matches_oracle_on_random_settings():
    # property test over (num_buckets, max_distance, direction): the library's host table (glibc
    # logf, float32 chain) and the oracle (the reference's torch expression) agree bit for bit
    from hypothesis import given, settings, strategies as st
    import turbot5_b200 as t5b
    from oracle import t5_oracle as orc

    @settings(max_examples=150, deadline=None)
    @given(st.sampled_from([4, 6, 8, 12, 16, 24, 32, 40, 64, 96, 128, 256]), st.integers(2, 2048), st.booleans())
    def check(nb, md, bidir):
        n_side = nb // 2 if bidir else nb
        if n_side < 2 or md <= n_side // 2:
            with pytest.raises(RuntimeError):
                t5b.relative_position_bucket_table(nb, md, bidir)
            return
        got = t5b.relative_position_bucket_table(nb, md, bidir, -md - 3, md + 3).numpy()
        want = orc.bucket_of_delta(range(-md - 3, md + 4), bidir, nb, md)
        assert np.array_equal(got, want), (nb, md, bidir)
        # monotone in distance on each side and saturating at max_distance
        neg = got[:md + 4][::-1]
        assert np.all(np.diff(neg) >= 0) and neg[md] == neg[-1]
    check()


def test_attention_workspace_query_is_zero_without_a_device_or_when_not_applicable():
    from turbot5_b200 import _native as nat
    L = nat.lib()
    a = nat.AttnArgs()
    assert L.t5b_attention_workspace_bytes(None) == 0
    a.dtype, a.D, a.B, a.H, a.M, a.N = nat.F32, 64, 1, 1, 4096, 4096
    assert L.t5b_attention_workspace_bytes(a) == 0        # float32 never takes the tensor-core kernel


def test_hot_kernels_stay_within_their_register_and_spill_budget():
    """ptxas's own report for the tensor-core kernels of the bench workload (bf16, head dim 64, no window):
    two blocks per SM need <= 96 registers, and the softmax loops are written to (almost) fit in them.
    Extra loop-live values show up here as spills long before any numerical test notices."""
    from turbot5_b200 import build
    fwd = build.resource_report("attn_fwd_sm100.cu")
    bwd = build.resource_report("attn_bwd_sm100.cu")

    def pick(report, *parts):
        names = [n for n in report if all(p in n for p in parts)]
        assert len(names) == 1, (parts, names)
        return report[names[0]]
    # mangled template arguments: Lb1 = bf16, Li64 = head dim, Li0 = no FMA-pipe exponentials, then Lb0 = no
    # window and Lb0 / Lb1 = head dim 64 itself / the kernel that also takes head dims 16 and 32
    for narrow in ("Lb0E", "Lb1E"):
        k = pick(fwd, "attn_fwd_kernel", "ILb1ELi64ELi0ELb0E" + narrow)
        assert k["registers"] <= 96 and k["spill_stores"] <= 128, k
    k = pick(bwd, "attn_bwd_dq_kernel", "ILb1ELi64ELb0E")
    assert k["registers"] <= 96 and k["spill_stores"] <= 16, k
    k = pick(bwd, "attn_bwd_dkv_wide_kernel", "ILb1ELb0E")
    assert k["registers"] <= 96 and k["spill_stores"] <= 64, k


def test_decoder_step_takes_every_documented_size():
    """One plan of tiles serves the size check and the launches, so a size that is accepted is one that runs: every
    documented width at every kind of batch, and nothing beyond."""
    import ctypes as C
    from turbot5_b200 import _native as nat
    P, I = C.c_void_p, C.c_int32

    class Args(C.Structure):
        _fields_ = [(n, P) for n in ("layers", "final_ln", "lm_head", "embedding", "table", "hidden", "logits", "tokens", "seqlens",
                                     "enc_seqlens", "workspace")] + \
                   [(n, C.c_int64) for n in ("workspace_bytes", "tokens_stride", "table_stride0", "cross_stride_b", "cross_stride_h",
                                             "cross_stride_n")] + \
                   [(n, I) for n in ("dtype", "table_dtype", "n_layers", "B", "H", "D", "d_model", "d_ff", "gated", "vocab", "max_len",
                                     "enc_len", "num_buckets", "max_distance")] + \
                   [("eps", C.c_float), ("lm_scale", C.c_float), ("device_status", P)]
    size = nat.lib().t5b_decoder_step_workspace_bytes
    size.restype, size.argtypes = C.c_int64, [P]

    def taken(dtype=nat.BF16, B=16, H=12, D=64, d_model=768, d_ff=2048, gated=1, max_distance=128):
        a = Args(dtype=dtype, table_dtype=dtype, n_layers=1, B=B, H=H, D=D, d_model=d_model, d_ff=d_ff, gated=gated, vocab=32128,
                 max_len=64, enc_len=512, num_buckets=32, max_distance=max_distance)
        return size(C.byref(a)) > 0
    for dtype in (nat.BF16, nat.F16):
        for B in (1, 2, 16, 17, 32, 33, 48, 64):
            for d_model in range(32, 2049, 32):
                assert taken(dtype, B, d_model=d_model), (dtype, B, d_model)
                assert taken(dtype, B, H=64, d_model=d_model, d_ff=8192), (dtype, B, d_model)
        for gated in (0, 1):
            for d_ff in range(32, 8193, 32):
                assert taken(dtype, d_model=2048, H=32, d_ff=d_ff, gated=gated), (dtype, d_ff, gated)
        for H, D in ((1, 32), (2, 16), (64, 64), (32, 128), (33, 64), (256, 16)):
            assert taken(dtype, H=H, D=D)
    for bad in (dict(B=65), dict(B=0), dict(d_model=2080), dict(d_model=40), dict(d_ff=8224), dict(H=65), dict(D=48), dict(dtype=nat.F32),
                dict(max_distance=2049)):
        assert not taken(**bad), bad


def test_whole_numbers_beyond_64_bits_raise_at_the_binding():
    import turbot5_b200 as t5b
    q = torch.zeros(1, 1, 4, 16)
    for kw in (dict(NUM_BUCKETS=1 << 70), dict(MAX_DISTANCE=-(1 << 70)), dict(q_pos_offset=1 << 64)):
        with pytest.raises(OverflowError):
            t5b.flash_attention_with_fusing_bias(q, q, q, None, **kw)
    with pytest.raises(RuntimeError):
        t5b.flash_attention_with_fusing_bias(q, q, q, None, q_pos_offset=-1)     # (there is no CPU path)


def test_norm_backward_keeps_two_blocks_per_sm():
    """256 threads and two blocks per SM need 128 registers at most: at d = 768 the residual's vectors would cost the
    second block, so the call without a residual has a kernel of its own (template arguments: type, weight type,
    columns / 256, residual)."""
    from turbot5_b200 import build
    report = build.resource_report("rmsnorm.cu")
    for t in ("13__nv_bfloat16", "6__half"):
        for variant in ("Li2ELb0E", "Li2ELb1E", "Li3ELb0E"):
            names = [n for n in report if "rmsnorm_bwd_vec_kernelI" + t in n and variant in n]
            assert len(names) == 1, (t, variant)
            k = report[names[0]]
            assert k["registers"] <= 128 and k["spill_stores"] == 0, (names[0], k)


def test_forward_kernels_of_every_form_of_call_stay_within_their_budget():
    """The forms that serve most calls (dense causal, dense whole, packed, block-local): 96 registers for two blocks per
    SM, and next to no spills (the kernels with the merge of a split wave have 48-92 bytes outside the loop)."""
    from turbot5_b200 import build
    report = build.resource_report("attn_fwd_sm100.cu")
    forms = {n: k for n, k in report.items() if "attn_fwd_case_kernel" in n}
    assert len(forms) == 2 * 2 * 4          # types, head dims, forms
    for n, k in forms.items():
        assert k["registers"] <= 96 and k["spill_stores"] <= 24, (n, k)
