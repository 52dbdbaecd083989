"""CPU-only checks of the boundary: the library loads, exports every declared symbol, and rejects bad calls on the
host before anything would be launched. No compute call is made here."""
import ctypes
import re
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def L():
    from pragnosia_b200 import build, _lib
    build.build()
    return _lib.lib()


def declared_symbols():
    text = (ROOT / "include" / "pragnosia_b200.h").read_text()
    return sorted(set(re.findall(r"^(?:int|long long|const char \*)\s*(pgb_[a-z0-9_]+)\(", text, flags=re.M)))


def test_every_declared_symbol_is_exported(L):
    names = declared_symbols()
    assert len(names) >= 9
    for n in names:
        assert hasattr(L, n), f"{n} declared in include/pragnosia_b200.h but not exported"


def test_binding_table_matches_header(L):
    from pragnosia_b200 import _lib
    header = set(declared_symbols()) - {"pgb_status_string", "pgb_last_cuda_error"}
    assert set(_lib.SIGNATURES) == header


def test_status_strings(L):
    assert L.pgb_abi_version() == 1
    assert L.pgb_status_string(0) == b"ok"
    assert b"NULL" in L.pgb_status_string(1)


def test_bad_calls_are_rejected_on_the_host(L):
    one = ctypes.c_void_p(0x1000)        # a non-null, 16-byte aligned, never dereferenced address
    odd = ctypes.c_void_p(0x1004)
    # null pointers
    assert L.pgb_lambda_scan_fwd(None, one, one, 0, 0, None, None, one, one, one, 1, 1, 4, None) == 1
    # state given only half
    assert L.pgb_lambda_scan_fwd(one, one, one, 0, 0, one, None, one, one, one, 1, 1, 4, None) == 1
    # bad shape
    assert L.pgb_lambda_scan_fwd(one, one, one, 0, 0, None, None, one, one, one, 0, 1, 4, None) == 2
    assert L.pgb_lambda_scan_fwd_ex(one, one, one, 0, 0, None, None, one, one, one, 1, 1, 4, 3, None) == 2
    # unsupported head dim, dtype, precision, alignment in the prefill
    args = lambda D=64, dt=0, prec=0, q=one: (q, one, one, dt, one, None, None, None, None, 0.0, one, dt, one, None, 1, 1, 8, D, prec, None)
    assert L.pgb_aspin_prefill_fwd(*args(D=96)) == 3
    assert L.pgb_aspin_prefill_fwd(*args(dt=7)) == 5
    assert L.pgb_aspin_prefill_fwd(*args(prec=9)) == 2
    assert L.pgb_aspin_prefill_fwd(*args(q=odd)) == 4
    # prep: stride that breaks the per-lane vector alignment
    assert L.pgb_aspin_prep_fwd(one, one, one, 0, 7, 7, 7, None, 0, 0, one, one, one, one, one, 1, 1, 4, 2, 64, None) == 4
    assert L.pgb_aspin_prep_fwd(one, one, one, 0, 512, 128, 64, None, 0, 0, one, one, one, one, one, 1, 1, 4, 2, 32, None) == 3
    # decode: the delta rule without beta; batch stride smaller than a row
    dec = lambda gate=None, delta=0, sb=64: (one, one, one, 0, sb, 1, gate, 1, 1, delta, one, 1, None, one, None, 0.0, one, one,
                                             None, 0.0, one, 0, 64, 1, 1, 64, None)
    assert L.pgb_aspin_decode_step(*dec(delta=1)) == 1
    assert L.pgb_aspin_decode_step(*dec(sb=8)) == 2
    assert L.pgb_rotate_pairs(one, 0, one, one, one, 1, 1, 1, 7, None) == 2
    # fused small-batch linear: norm without its weight, more than eight rows, K not a multiple of 8, unaligned W
    sk = lambda nw=None, kind=0, B=1, K=768, W=one: (one, None, nw, None, kind, 1e-5, W, None, 0, one, None, B, K, 16, None)
    assert L.pgb_skinny_linear(*sk(kind=1)) == 1
    assert L.pgb_skinny_linear(*sk(B=9)) == 7
    assert L.pgb_skinny_linear(*sk(K=100)) == 2
    assert L.pgb_skinny_linear(*sk(W=odd)) == 4
    # decode-step ends: d not a multiple of 8; a negative temperature; a missing ticket
    assert L.pgb_decode_embed(one, one, one, one, one, 1, 60, 10, 10, None) == 2
    assert L.pgb_decode_sample(one, 0, -1.0, 0, one, None, 0, one, None, None, one, 1, 8, 1, None) == 2
    assert L.pgb_decode_sample(one, 0, 1.0, 0, one, None, 0, one, None, None, None, 1, 8, 1, None) == 1


def test_ops_refuse_cpu_tensors():
    from pragnosia_b200 import ops
    x = torch.zeros(1, 4, 8)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.lambda_scan(x, x, x)
    q = torch.zeros(1, 1, 8, 64)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.prefill(q, q, q, torch.zeros(1, 1, 8))


def test_model_loads_reference_named_checkpoints():
    """The modules keep the reference's parameter names and shapes, so its state_dicts load strictly."""
    import oracle
    from pragnosia_b200.model import LM
    for mixer, norm in (("aspin", "ln"), ("dspin", "rms"), ("hspin", "ln"), ("hdspin", "rms"), ("fspin", "ln")):
        cfg = oracle.lm_config(256, 128, 2, 2, 32, mixer, norm)
        m = LM(256, 128, 2, 2, 32, mixer, norm)
        m.load_state_dict(oracle.init_lm_params(cfg, 0), strict=True)
    n = sum(p.numel() for p in LM().parameters())
    assert abs(n / 1e6 - 91.93) < 0.01
    with pytest.raises(NotImplementedError):
        LM(mixer="attn")


def test_lambda_scan_segment_choice(L):
    """The host picks more time segments when there are few channels and never more than the sequence has pieces."""
    ts = lambda B, T, D: L.pgb_lambda_scan_time_segments(B, T, D, 148)
    assert ts(64, 32768, 768) == 8                             # 12288 channel quads x 8 segments: whole rounds of resident warps
    assert ts(1, 32768, 64) == 32                              # 16 quads: the time axis must supply the parallelism
    assert ts(1, 32768, 64) >= ts(8, 32768, 768) >= ts(64, 32768, 768)
    assert ts(2, 1, 300) == 1 and ts(2, 6, 300) <= 2           # a short sequence has nothing to split
    for B, T, D in ((2, 45, 300), (16, 512, 704), (3, 1000, 24)):
        t = ts(B, T, D)
        assert t in (1, 2, 4, 8, 16, 32)
    assert ts(0, 5, 5) == 0 and L.pgb_lambda_scan_time_segments(1, 5, 5, 0) == 0


def test_new_entry_points_reject_bad_calls(L):
    one = ctypes.c_void_p(0x1000)
    assert L.pgb_assoc_out_fwd(one, one, one, 0, one, None, one, 1, 1, 8, 64, None) == 1
    assert L.pgb_assoc_out_fwd(one, one, one, 0, one, one, one, 1, 1, 8, 96, None) == 3
    assert L.pgb_prefix_scan_fwd(one, one, 9, one, one, None, one, one, 1, 1, 1, 64, None) == 5
    assert L.pgb_delta_inv_fwd(ctypes.c_void_p(0x1004), one, one, one, 1, 1, 8, 64, None) == 4
    assert L.pgb_delta_loop_fwd(one, one, 0, one, None, one, None, one, one, one, 1, 1, 8, 64, None) == 1
    assert L.pgb_key_topk_mask(one, 0, 64, 64, 64, 1, 1, 1, 64, 0, None) == 2
    assert L.pgb_key_topk_mask(one, 0, 64, 64, 64, 1, 1, 1, 64, 65, None) == 2
    assert L.pgb_short_conv_fwd(one, 0, 8, 8, one, one, one, one, 1, 1, 8, 4, None) == 2       # cache_in == cache_out
    assert L.pgb_lambda_scan_bwd(one, one, one, one, 0, 0, one, None, None, one, one, one, None, None, 1, 1, 4, None) == 1
    assert L.pgb_lambda_scan_bwd(one, one, one, one, 0, 0, one, one, None, one, one, one, one, None, 1, 1, 4, None) == 1
    assert L.pgb_aspin_prep_bwd(one, one, one, 0, 64, 64, 64, one, 1, 1, one, one, one, one, one, 0, one, one, one, None, one,
                                1, 1, 1, 64, None) == 1                                          # a gate without room for its gradient
    assert L.pgb_decode_sample_ex(one, 0, 1.0, 1.5, 0, one, None, 0, one, None, None, one, 1, 8, 1, None) == 2
    assert L.pgb_skinny_linear_ex(one, None, None, None, 0, 1e-5, one, None, 0, one, None, 1, 768, 16, 4, None) == 2
    assert L.pgb_aspin_prep_bwd_tiles(17) == 3
    # the plain rule's two backward kernels, the batch linear layer
    assert L.pgb_assoc_out_bwd(one, one, one, 0, one, one, one, one, one, one, one, None, 1, 1, 8, 64, None) == 1
    assert L.pgb_assoc_out_bwd(one, one, one, 0, one, one, one, one, one, one, one, one, 1, 1, 8, 96, None) == 3
    assert L.pgb_prefix_scan_bwd(one, one, 7, one, one, one, None, None, one, one, one, one, None, 1, 1, 1, 64, None) == 5
    assert L.pgb_batch_linear(one, one, None, one, 129, 16, 64, 0, None) == 7 and L.pgb_batch_linear(one, one, None, one, 4, 12, 64, 0, None) == 2
    assert L.pgb_batch_linear_ex(one, one, one, one, 4, 16, 64, 0, one, 1, one, one, 1, 1e-5, None, None, 0, None) == 1   # folded norm + bias
    assert L.pgb_batch_linear_ex(one, one, None, one, 4, 16, 64, 0, None, 0, None, None, 0, 0.0, None, None, 2, None) == 2  # unknown flag
    assert L.pgb_batch_linear_parts(768) == 48
    assert L.pgb_decode_set_variant(3) == 2 and L.pgb_decode_set_variant(0) == 0
    assert L.pgb_linear_act_set_variant(6) == 2 and L.pgb_linear_act_set_variant(-1) == 2 and L.pgb_linear_act_set_variant(0) == 0
    # the one-launch decode step: scratch size, then the rejects (bias missing for a layer norm, short scratch, batch, head dim)
    assert L.pgb_decode_token_work_bytes(1, 768, 2328, 3072) == 2 * (4 * 768 + 2328 + 3072)
    tok = lambda **kw: L.pgb_decode_token_fwd(one, 12, one, one, one, kw.get("nb", one), 2, 1e-5, one, one, one, one, kw.get("wb", 10 ** 6),
                                              one, one, kw.get("B", 1), 768, 12, kw.get("D", 64), 2328, 3072, 50257, 512, 0, None)
    assert tok(nb=None) == 1 and tok(wb=10) == 2 and tok(B=5) == 7 and tok(D=96) == 3
    # the linear layers of a batch's step: which K they take, then the rejects (batch, a residual without its norm weight, both results, K too long)
    assert L.pgb_decode_linear_takes(0, 2328, 768) == 1 and L.pgb_decode_linear_takes(1, 768, 768 * 16) == 0 and L.pgb_decode_linear_takes(0, 12, 768) == 0
    assert L.pgb_decode_linear_parts(768, 768, 64) == 24 and L.pgb_decode_linear_parts(768, 256, 8) == 48 and L.pgb_decode_linear_parts(768, 192, 8) == 0
    assert L.pgb_decode_linear_parts(768, 3072, 32) == 16 and L.pgb_decode_linear_parts(768, 3072, 33) == 24
    lin = lambda **kw: L.pgb_decode_linear(one, one, one, None, 0, 0.0, 0, kw.get("resid"), kw.get("next_w"), kw.get("y", one), kw.get("yw"), kw.get("sq"),
                                           kw.get("logits"), None, None, kw.get("window", 0), kw.get("B", 4), 768, kw.get("K", 768), None)
    assert lin(B=65) == 7 and lin(K=768 * 16) == 7 and lin(K=12) == 2 and lin(resid=one) == 1 and lin(logits=one) == 1 and lin(y=None) == 1
    assert lin(window=512) == 1 and lin(y=ctypes.c_void_p(0x1004)) == 4
    assert L.pgb_decode_embed_norm(one, one, one, one, None, one, one, one, 4, 768, 100, 16, None) == 1
    # delta rule: scratch beyond the inverses where few chains at head dim 64 are walked in segments side by side, never more than 256 MiB of it
    x, more = L.pgb_aspin_delta_scratch_bytes, L.pgb_aspin_delta_prefill_scratch_bytes
    assert more(3, 12, 1333, 64) > x(3, 12, 1333) and more(1, 2, 2048, 64) > x(1, 2, 2048) and more(3, 12, 1333, 128) == x(3, 12, 1333)
    assert more(8, 16, 8192, 64) == x(8, 16, 8192) and more(1, 2, 128, 64) == x(1, 2, 128) and more(1, 1, 1 << 22, 64) == x(1, 1, 1 << 22)
    assert 0 <= L.pgb_aspin_delta_layer_scratch_bytes(3, 12, 1333, 64) - L.pgb_aspin_delta_layer_scratch_least_bytes(3, 12, 1333, 64) <= 256 << 20
    # the same step without barriers: 32-bit words of every layer's exchanges; 0 where a row does not fit a stage or the rows shared memory
    assert L.pgb_decode_flow_work_bytes(12, 2, 768, 2328, 3072) == 4 * 12 * 2 * (2328 + 3 * 768 + 3072)
    assert L.pgb_decode_flow_work_bytes(12, 1, 3200, 9624, 12800) == 0 and L.pgb_decode_flow_work_bytes(12, 4, 2048, 6208, 8192) == 0
    assert L.pgb_decode_flow_work_bytes(12, 5, 768, 2328, 3072) == 0 and L.pgb_decode_flow_work_bytes(0, 1, 768, 2328, 3072) == 0
    flow = lambda **kw: L.pgb_decode_flow_step_fwd(one, 12, one, one, one, kw.get("nb", one), 2, 1e-5, one, one, one, 512, kw.get("work", one),
                                                   kw.get("wb", 10 ** 6), one, one, kw.get("B", 1), 768, 12, kw.get("D", 64), 2328, 3072, 50257, 512, 0, None)
    assert flow(nb=None) == 1 and flow(wb=10) == 2 and flow(B=5) == 7 and flow(D=96) == 3 and flow(work=ctypes.c_void_p(0x1008)) == 4


def test_segments_and_windows_refuse_an_in_place_state(L):
    """Their CTAs run side by side: one would write the state that another has yet to read."""
    one, st = ctypes.c_void_p(0x1000), ctypes.c_void_p(0x2000)
    n = L.pgb_aspin_prefill_segments_scratch_bytes(1, 1, 4096, 64)
    assert n > 0
    seg = lambda S0, S: L.pgb_aspin_prefill_segments_fwd(one, one, one, one, S0, None, None, 0.0, one, 1, S, None, one, n, 1, 1, 4096, 64, None)
    assert seg(st, st) == 2
    win = lambda S0, S: L.pgb_aspin_layer_prefill_windows_ex(one, one, one, 4096, 64, one, one, 4096, 64, one, one, 64, one, S0, one, 1e-5, one, S, one,
                                                             1 << 30, 64, 1, 1, 128, 64, None)
    assert win(st, st) == 2
    delta = lambda S0, S: L.pgb_aspin_delta_layer_windows_ex(one, one, one, 4096, 64, one, one, 4096, 64, one, one, one, S0, one, 1e-5, one, S, one,
                                                             1 << 30, 64, 1, 1, 128, 64, None)
    assert delta(st, st) == 2


def test_variants_as_one_number(L):
    assert L.pgb_variants() == 0
    assert L.pgb_tc_set_variant(1) == 0 and L.pgb_linear_act_set_variant(3) == 0 and L.pgb_decode_set_variant(2) == 0
    assert L.pgb_variants() == 1 + (3 << 4) + (2 << 12)
    assert L.pgb_tc_set_variant(0) == 0 and L.pgb_linear_act_set_variant(0) == 0 and L.pgb_decode_set_variant(0) == 0
    assert L.pgb_variants() == 0


def test_bench_table_names_are_kernel_bench_cases():
    """bench.py's per-kernel table is built from kernel_bench cases by name: every name it asks for exists."""
    import ast
    import pathlib
    from pragnosia_b200 import kernel_bench as kb
    src = (pathlib.Path(__file__).resolve().parents[1] / "bench.py").read_text()
    fn = next(n for n in ast.walk(ast.parse(src)) if isinstance(n, ast.FunctionDef) and n.name == "kernel_rooflines")
    names = [c.value for t in ast.walk(fn) if isinstance(t, ast.Tuple) for c in t.elts if isinstance(c, ast.Constant) and isinstance(c.value, str)]
    asked = [n for n in names if n in kb.CASES or n.startswith(("prefill", "decode", "lambda", "layer_"))]
    assert len(asked) >= 15 and all(n in kb.CASES for n in asked), [n for n in asked if n not in kb.CASES]
    assert all(n in kb.CASES for n in kb.FLOPS)


def test_linear_layers_of_a_batchs_step_are_taken_at_every_batch_or_at_none(L):
    """pgb_decode_linear_takes knows no batch: what it accepts, pgb_decode_linear and pgb_decode_linear_parts accept at every batch up to 64, and what it
    refuses they refuse. x misaligned: a call whose sizes are accepted ends at that check (4), so none is launched; 7 is a refused size."""
    one, odd = ctypes.c_void_p(0x1000), ctypes.c_void_p(0x1004)
    taken = 0
    for K in (*range(8, 1024, 8), *range(1024, 17408, 64)):
        for kind in range(3):
            takes = L.pgb_decode_linear_takes(kind, 768, K)
            taken += takes
            for B in range(1, 65):
                r, lg = (one if kind == 1 else None), (one if kind == 2 else None)
                rc = L.pgb_decode_linear(odd, one, None, None, 0, 0.0, 0, r, r, None if lg else one, r, r, lg, None, None, 0, B, 768, K, None)
                assert rc == (4 if takes else 7), (kind, K, B)
                if kind == 1:
                    assert (L.pgb_decode_linear_parts(768, K, B) > 0) == bool(takes), (K, B)
    assert taken > 0 and L.pgb_decode_linear_takes(1, 1792, 7168) == 1


def test_wrappers_of_the_chained_step_see_lengths():
    """The kernels read bias, norm weights and tables to the sizes of x and W, and the C entry points see addresses only: a tensor that is too short, of
    another width or not laid out row by row is refused by the wrapper, ahead of the check for the device that right ones end at here."""
    from pragnosia_b200 import ops
    bf = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    B, N, K = 5, 24, 256
    lin = lambda **kw: ops.decode_linear(kw.pop("x", bf(B, K)), kw.pop("W", bf(N, K)), kw.pop("bias", bf(N)), **kw)
    long, f32 = (lambda n: torch.zeros(n, dtype=torch.long)), torch.zeros
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        lin(squares=f32(B, 3), resid=bf(B, N), next_w=bf(N))
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        lin(logits=f32(B, N), pos=long(1), shift=f32(()), window=8)
    for bad in (dict(bias=bf(N - 2)), dict(bias=bf(1, N)), dict(resid=bf(B, N), next_w=bf(N - 8)), dict(resid=bf(B, N - 8), next_w=bf(N)), dict(resid=bf(B, N)),
                dict(W=bf(N * K)), dict(squares=f32(B)), dict(squares=f32(B, 0)), dict(squares=f32(B - 1, 3)), dict(logits=f32(B, N), window=8),
                dict(logits=f32(B, N), pos=long(0), shift=f32(()), window=8), dict(logits=f32(B, N), pos=long(1), shift=f32(0), window=8)):
        with pytest.raises(ValueError):
            lin(**bad)
    emb = lambda **kw: ops.decode_embed_norm(long(B), kw.pop("pos", long(1)), kw.pop("E", bf(64, K)), kw.pop("P", bf(16, K)), kw.pop("w", bf(K)))
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        emb()
    for bad in (dict(pos=long(0)), dict(E=bf(K, 64).T), dict(P=bf(16, K - 8)), dict(P=bf(K, 16).T), dict(w=bf(K - 8)), dict(w=bf(2 * K)[::2])):
        with pytest.raises(ValueError):
            emb(**bad)
