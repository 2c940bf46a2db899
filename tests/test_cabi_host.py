"""Host-side behaviour of the C ABI and of the PersistentKernel mirror: the library
loads and exports every declared symbol, the lowering fuses what it may, and the
error behaviour follows the reference API.  No GPU, no compute calls."""
import ctypes as C
import os
import re

import pytest
import torch

import fleet_chiplet_megakernel_b200 as mk
from fleet_chiplet_megakernel_b200 import _cabi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol(native_lib):
    header = open(os.path.join(ROOT, "include", "b200mk.h")).read()
    declared = set(re.findall(r"\b(mk_[a-z_]+)\s*\(", header))
    assert declared, "no declarations found"
    for name in sorted(declared):
        assert hasattr(native_lib, name), f"{name} is declared but not exported"
    assert declared == set(_cabi.SIGNATURES), declared ^ set(_cabi.SIGNATURES)


@pytest.mark.parametrize("nblk,nkt,grid", [(48, 64, 148), (32, 64, 148), (192, 64, 148), (32, 192, 148),
                                           (1187, 64, 148), (1, 1, 148), (3, 5, 7), (148, 1, 148), (5, 2, 148)])
def test_tile_partition_is_a_contiguous_cover(native_lib, nblk, nkt, grid):
    begin = (C.c_int64 * (grid + 1))()
    bad = C.c_int(0)
    assert native_lib.mk_debug_partition(nblk, nkt, grid, begin, C.byref(bad)) == 0
    b = list(begin)
    assert b[0] == 0 and b[-1] == nblk * nkt and all(x <= y for x, y in zip(b, b[1:]))
    assert max(y - x for x, y in zip(b, b[1:])) - min(y - x for x, y in zip(b, b[1:])) <= 1
    assert bad.value == 0, "tile_owner disagrees with the ranges"


def _meta(R, T, max_seq, max_pages):
    return {
        "step": torch.zeros(R, dtype=torch.int32), "tokens": torch.zeros(R, max_seq, dtype=torch.int64),
        "input_tokens": torch.zeros(T, 1, dtype=torch.int64), "output_tokens": torch.zeros(T, 1, dtype=torch.int64),
        "num_new_tokens": torch.ones(R, dtype=torch.int32), "prompt_lengths": torch.ones(R, dtype=torch.int32),
        "qo_indptr_buffer": torch.zeros(R + 1, dtype=torch.int32),
        "paged_kv_indptr_buffer": torch.zeros(R + 1, dtype=torch.int32),
        "paged_kv_indices_buffer": torch.zeros(max_pages, dtype=torch.int32),
        "paged_kv_last_page_len_buffer": torch.zeros(R, dtype=torch.int32),
    }


def _kernel(mode="offline", R=2, max_seq=64, page=16, pages=8, **kw):
    return mk.PersistentKernel(mode=mode, world_size=1, mpi_rank=0, num_workers=0, num_local_schedulers=0,
                               num_remote_schedulers=0, max_seq_length=max_seq, max_num_batched_requests=R,
                               max_num_batched_tokens=R, max_num_pages=pages, page_size=page,
                               meta_tensors=_meta(R, R, max_seq, pages), profiler_tensor=None, trace_name="",
                               spec_decode_config=None, use_cutlass_kernel=True, **kw)


def _tiny_graph(k, layers=2):
    geom = mk.Qwen3Geometry(hidden=512, n_q=4, n_kv=2, mlp=1024, layers=layers, vocab=2048)
    w = {"embed": torch.zeros(geom.vocab, geom.hidden, dtype=torch.bfloat16),
         "lm_head": torch.zeros(geom.vocab, geom.hidden, dtype=torch.bfloat16),
         "norm": torch.ones(geom.hidden, dtype=torch.bfloat16)}
    for i in range(layers):
        w[f"l{i}.q"] = torch.zeros(geom.n_q * 128, geom.hidden, dtype=torch.bfloat16)
        w[f"l{i}.k"] = torch.zeros(geom.n_kv * 128, geom.hidden, dtype=torch.bfloat16)
        w[f"l{i}.v"] = torch.zeros(geom.n_kv * 128, geom.hidden, dtype=torch.bfloat16)
        w[f"l{i}.o"] = torch.zeros(geom.hidden, geom.n_q * 128, dtype=torch.bfloat16)
        w[f"l{i}.gate"] = torch.zeros(geom.mlp, geom.hidden, dtype=torch.bfloat16)
        w[f"l{i}.up"] = torch.zeros(geom.mlp, geom.hidden, dtype=torch.bfloat16)
        w[f"l{i}.down"] = torch.zeros(geom.hidden, geom.mlp, dtype=torch.bfloat16)
        for n, d in (("ln1", geom.hidden), ("ln2", geom.hidden), ("qn", 128), ("kn", 128)):
            w[f"l{i}.{n}"] = torch.ones(d, dtype=torch.bfloat16)
    kc = torch.zeros(layers, k.max_num_pages, k.page_size, geom.n_kv, 128, dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    cos = torch.zeros(k.max_seq_length, 128, dtype=torch.bfloat16)
    mk.build_qwen3_graph(k, geom, w, kc, vc, cos, cos.clone(), k.meta_tensors["input_tokens"],
                         k.meta_tensors["output_tokens"])
    return w, kc, vc, cos


def test_lowering_fuses_norm_silu_and_argmax(native_lib):
    k = _kernel(fuse=True)
    keep = _tiny_graph(k, layers=2)
    plan = k.plan().strip().splitlines()
    kinds = [ln.split()[1] for ln in plan]
    assert kinds == ["embed"] + ["linear", "attention", "linear", "linear", "linear"] * 2 + ["linear", "argmax_reduce"]
    assert sum("rmsnorm fused" in ln for ln in plan) == 5
    assert sum("silu_mul fused" in ln for ln in plan) == 2
    assert sum("argmax partials fused" in ln for ln in plan) == 1
    k.finalize()
    del keep


def test_lowering_without_fusion_keeps_every_layer(native_lib):
    k = _kernel(fuse=False)
    keep = _tiny_graph(k, layers=2)
    kinds = [ln.split()[1] for ln in k.plan().strip().splitlines()]
    per_layer = ["rmsnorm", "linear", "attention", "linear", "rmsnorm", "linear", "silu_mul", "linear"]
    assert kinds == ["embed"] + per_layer * 2 + ["rmsnorm", "linear", "argmax_partial", "argmax_reduce"]
    k.finalize()
    del keep


def test_error_behaviour_follows_the_reference_api(native_lib):
    with pytest.raises(ValueError, match="Invalid persistent kernel mode"):
        _kernel(mode="bogus")
    with pytest.raises(NotImplementedError, match="'online' is not built"):
        _kernel(mode="online")
    for one_pass in ("online_notoken", "onepass", "online_multi_turn"):  # one pass per call over the caller's metadata
        k = _kernel(mode=one_pass)
        assert k.mode == one_pass
        k.finalize()
    k = _kernel()
    with pytest.raises(RuntimeError, match="Invalid io_category"):
        k.new_tensor(dims=(2, 8), name="t", io_category="host_tensor")
    with pytest.raises(AssertionError):  # non row-major input, as the reference asserts
        k.attach_input(torch.zeros(8, 16, dtype=torch.bfloat16).t(), name="bad")
    with pytest.raises(AssertionError):  # a name is mandatory
        k.attach_input(torch.zeros(8, 16, dtype=torch.bfloat16))
    a = k.attach_input(torch.zeros(2, 64, dtype=torch.bfloat16), name="a")
    w = k.attach_input(torch.zeros(128, 32, dtype=torch.bfloat16), name="w")  # K mismatch
    o = k.new_tensor(dims=(2, 128), name="o")
    k.linear_layer(input=a, weight=w, output=o, grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    with pytest.raises(ValueError, match="K mismatch"):
        k.plan()
    k.finalize()
    k = _kernel()
    a = k.attach_input(torch.zeros(2, 64, dtype=torch.bfloat16), name="a")
    b = k.new_tensor(dims=(3, 2, 64), name="buf")
    o = k.new_tensor(dims=(2, 64), name="o")
    k.allreduce_layer(input=a, buffer=b, output=o, grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    assert "allreduce" in k.plan()  # planned; a single rank just copies
    k.finalize()
    k = _kernel()
    with pytest.raises(NotImplementedError, match="unknown layer"):
        k._op("sampling_sm100", [k.new_tensor(dims=(2, 64), name="z")])
        k.plan()
    k.finalize()


def test_lowering_picks_the_path_by_batch(native_lib):
    """One or two batched tokens fold the norms into the linears (row-owner path); more keep
    the rmsnorm tasks (activation boxes); page sizes must be powers of two."""
    for R, fused in ((1, 5), (2, 5), (3, 0), (16, 0)):
        k = _kernel(fuse=True, R=R, pages=R * 4)
        keep = _tiny_graph(k, layers=2)
        plan = k.plan().strip().splitlines()
        assert sum("rmsnorm fused" in ln for ln in plan) == fused, (R, plan)
        assert sum(ln.split()[1] == "rmsnorm" for ln in plan) == 5 - fused
        assert sum("silu_mul fused" in ln for ln in plan) == 2
        k.finalize()
        del keep
    k = _kernel(page=24, pages=8)
    keep = _tiny_graph(k, layers=1)
    with pytest.raises(NotImplementedError, match="power of two"):
        k.plan()
    k.finalize()
    del keep


@pytest.mark.skipif(torch.cuda.is_available(), reason="checks the no-GPU failure mode")
def test_compile_without_a_gpu_fails_loudly(native_lib):
    k = _kernel()
    keep = _tiny_graph(k, layers=1)
    with pytest.raises(RuntimeError, match="no CPU fallback"):
        k.compile()
    k.finalize()
    del keep


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_cabi, "_lib", None)
    monkeypatch.setattr(_cabi, "LIB_PATH", str(tmp_path / "libb200mk.so"))
    with pytest.raises(RuntimeError, match="no fallback"):
        _cabi.load()


# ---- the reference's other spellings of the same layers -------------------------------------
def _weights(geom, layers):
    z = lambda *sh: torch.zeros(*sh, dtype=torch.bfloat16)
    w = {"embed": z(geom.vocab, geom.hidden), "lm_head": z(geom.vocab, geom.hidden), "norm": z(geom.hidden)}
    for i in range(layers):
        w[f"l{i}.q"], w[f"l{i}.k"], w[f"l{i}.v"] = z(geom.n_q * 128, geom.hidden), z(geom.n_kv * 128, geom.hidden), z(geom.n_kv * 128, geom.hidden)
        w[f"l{i}.o"], w[f"l{i}.gate"], w[f"l{i}.up"] = z(geom.hidden, geom.n_q * 128), z(geom.mlp, geom.hidden), z(geom.mlp, geom.hidden)
        w[f"l{i}.down"] = z(geom.hidden, geom.mlp)
        for n, d in (("ln1", geom.hidden), ("ln2", geom.hidden), ("qn", 128), ("kn", 128)):
            w[f"l{i}.{n}"] = z(d)
    return w


def _variant_graph(k, variant, layers=2):
    """The layer-call sequence of the reference's model builder with its split-K projections
    (python/mirage/mpk/models/qwen3/builder.py:560-700, cc-100 branch: splitk_linear_layer
    accumulating into the residual stream) or of its driver with USE_GANG=1
    (demo/qwen3/demo.py:560-1170: gang_rmsnorm / gang_linear / gang attention / fused SiLU)."""
    geom = mk.Qwen3Geometry(hidden=512, n_q=4, n_kv=2, mlp=1024, layers=layers, vocab=2048)
    w = _weights(geom, layers)
    T, R, H, D = k.max_num_batched_tokens, k.max_num_batched_requests, geom.hidden, 128
    qkv_out = (geom.n_q + 2 * geom.n_kv) * D
    kc = torch.zeros(layers, k.max_num_pages, k.page_size, geom.n_kv, D, dtype=torch.bfloat16)
    vc = torch.zeros_like(kc)
    cos = torch.zeros(k.max_seq_length, D, dtype=torch.bfloat16)
    sin = cos.clone()
    keep = [w, kc, vc, cos, sin]
    gang = variant == "gang"
    x = k.attach_input(k.meta_tensors["input_tokens"], "input_token")
    cos_t, sin_t = k.attach_input(cos, "cos"), k.attach_input(sin, "sin")
    y = k.new_tensor(dims=(T, H), name="embed_out")
    rms = k.new_tensor(dims=(T, H), name="rmsnorm_out")
    attn_in = k.new_tensor(dims=(T, qkv_out), name="attn_in")
    attn_out = k.new_tensor(dims=(T, geom.n_q * D), name="attn_out")
    attn_proj = k.new_tensor(dims=(T, H), name="attn_proj_out")
    mlp_mid = k.new_tensor(dims=(T, 2 * geom.mlp), name="mlp_mid")
    silu_out = k.new_tensor(dims=(T, geom.mlp), name="silu_mul_out")
    mlp_out = k.new_tensor(dims=(T, H), name="mlp_out")
    chunks = 2
    if gang:
        lse = k.new_tensor(dims=(T, chunks * geom.n_q), dtype=mk.float32, name="lse")
        tmp = k.new_tensor(dims=(T, chunks * geom.n_q * D), name="attn_out_tmp")
        qws = k.new_tensor(dims=(T, geom.n_q * D), name="q_ws")
        ws = k.new_tensor(dims=(4 * T, H), dtype=mk.float32, name="splitk_ws")
    k.embed_layer(input=x, weight=k.attach_input(w["embed"], "embed"), output=y, grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    x = y
    for i in range(layers):
        wq, wk, wv = (k.attach_input(w[f"l{i}.{n}"], f"l{i}{n}") for n in "qkv")
        wqkv = k.shuffle_tensors([wq, wk, wv], 0, geom.n_kv, name=f"l{i}qkv")
        wn = k.attach_input(w[f"l{i}.ln1"], f"l{i}ln1")
        if gang:
            k.gang_rmsnorm_layer(input=x, weight=wn, output=rms)
            k.gang_linear_layer(input=rms, weight=wqkv, output=attn_in, tile_n=64, output_stride=qkv_out, m_tiles=1, wgm=0)
        else:
            k.rmsnorm_layer(input=x, weight=wn, output=rms, grid_dim=(T, 1, 1), block_dim=(128, 1, 1))
            k.linear_layer(input=rms, weight=wqkv, output=attn_in, grid_dim=(qkv_out // 64, 1, 1), block_dim=(128, 1, 1))
        qn, kn = k.attach_input(w[f"l{i}.qn"], f"l{i}qn"), k.attach_input(w[f"l{i}.kn"], f"l{i}kn")
        kct, vct = k.attach_input(kc[i], f"l{i}kc"), k.attach_input(vc[i], f"l{i}vc")
        if gang:
            k.gang_paged_attention_split_kv_layer(input=attn_in, k_cache=kct, v_cache=vct, q_norm=qn, k_norm=kn,
                                                  cos_pos_embed=cos_t, sin_pos_embed=sin_t, lse=lse, output=tmp,
                                                  q_workspace=qws, attention_params=(geom.n_q, chunks, geom.n_q * D),
                                                  block_dim=(256, 1, 1))
            k.gang_paged_attention_split_kv_merge_layer(lse=lse, output_tmp=tmp, output=attn_out,
                                                        attention_params=(geom.n_q, D, geom.n_kv, chunks), block_dim=(256, 1, 1))
        else:
            k.paged_attention_layer(input=attn_in, k_cache=kct, v_cache=vct, q_norm=qn, k_norm=kn, cos_pos_embed=cos_t,
                                    sin_pos_embed=sin_t, output=attn_out, grid_dim=(R, geom.n_kv, 1), block_dim=(128, 1, 1))
        wo = k.attach_input(w[f"l{i}.o"], f"l{i}o")
        if variant == "splitk":
            k.splitk_linear_layer(input=attn_out, weight=wo, output=x, grid_dim=(H // 128, 128 * 128 // H, 1), block_dim=(256, 1, 1))
        elif gang:
            k.gang_linear_with_residual_layer(input=attn_out, weight=wo, residual=x, output=attn_proj, tile_n=64, output_stride=H)
            x = attn_proj
        else:
            k.linear_with_residual_layer(input=attn_out, weight=wo, residual=x, output=attn_proj, grid_dim=(H // 64, 1, 1), block_dim=(128, 1, 1))
            x = attn_proj
        wg, wu = k.attach_input(w[f"l{i}.gate"], f"l{i}g"), k.attach_input(w[f"l{i}.up"], f"l{i}u")
        tasks = 2 * geom.mlp // 64
        wgu = k.shuffle_tensors([wg, wu], 0, tasks // 2, name=f"l{i}gu")
        wn2 = k.attach_input(w[f"l{i}.ln2"], f"l{i}ln2")
        wd = k.attach_input(w[f"l{i}.down"], f"l{i}d")
        if gang:
            k.gang_rmsnorm_layer(input=x, weight=wn2, output=rms)
            k.gang_linear_silu_layer(input=rms, weight=wgu, output=silu_out, tile_n=64, output_stride=geom.mlp)
            k.gang_splitk_linear_with_residual_layer(input=silu_out, weight=wd, residual=x, workspace=ws, output=mlp_out,
                                                     tile_n=64, output_stride=H, k_splits=4)
            x = mlp_out
        else:
            k.rmsnorm_layer(input=x, weight=wn2, output=rms, grid_dim=(T, 1, 1), block_dim=(128, 1, 1))
            k.linear_layer(input=rms, weight=wgu, output=mlp_mid, grid_dim=(tasks, 1, 1), block_dim=(128, 1, 1))
            k.silu_mul_layer(input=mlp_mid, output=silu_out, grid_dim=(tasks // 2, 1, 1), block_dim=(128, 1, 1))
            if variant == "splitk":
                k.splitk_linear_layer(input=silu_out, weight=wd, output=x, grid_dim=(H // 128, 128 * 128 // H, 1), block_dim=(256, 1, 1))
            else:
                k.linear_with_residual_layer(input=silu_out, weight=wd, residual=x, output=mlp_out, grid_dim=(H // 64, 1, 1), block_dim=(128, 1, 1))
                x = mlp_out
    return keep


def _shape_of(plan):
    """(kind, n, k, flags) per device op: what the program does, independent of tensor names."""
    out = []
    for ln in plan.strip().splitlines():
        f = ln.split()
        kv = dict(x.split("=", 1) for x in f[2:] if "=" in x)
        out.append((f[1], kv["n"], kv["k"], kv["flags"]))
    return out


@pytest.mark.parametrize("R", [1, 4])
def test_split_k_and_gang_spellings_lower_to_the_plain_program(native_lib, R):
    plans = {}
    for variant in ("plain", "splitk", "gang"):
        k = _kernel(R=R, pages=4 * R, fuse=True)
        keep = _variant_graph(k, variant)
        plans[variant] = k.plan()
        k.finalize()
        del keep
    base = _shape_of(plans["plain"])
    assert [b[0] for b in base] == ["embed"] + (["linear", "attention", "linear", "linear", "linear"] if R <= 2 else
                                                ["rmsnorm", "linear", "attention", "linear", "rmsnorm", "linear", "linear"]) * 2
    assert _shape_of(plans["splitk"]) == base
    assert _shape_of(plans["gang"]) == base
    assert plans["splitk"].count("accumulates into its output") == 4


def test_fused_silu_linear_and_workspace_split_k(native_lib):
    k = _kernel(R=4, pages=16)
    T = 4
    x = k.attach_input(torch.zeros(T, 256, dtype=torch.bfloat16), "x")
    g, u = k.attach_input(torch.zeros(512, 256, dtype=torch.bfloat16), "g"), k.attach_input(torch.zeros(512, 256, dtype=torch.bfloat16), "u")
    wgu = k.shuffle_tensors([g, u], 0, 1, name="gu")
    mid = k.new_tensor(dims=(T, 1024), name="mid")
    wd = k.attach_input(torch.zeros(256, 512, dtype=torch.bfloat16), "wd")
    ws = k.new_tensor(dims=(2 * T, 256), name="ws")
    o1, o2 = k.new_tensor(dims=(T, 256), name="o1"), k.new_tensor(dims=(T, 256), name="o2")
    k.linear_layer(input=x, weight=wgu, output=mid, grid_dim=(8, 1, 1), block_dim=(128, 1, 1))
    k.silu_mul_linear_with_residual_layer(input=mid, weight=wd, residual=x, output=o1, grid_dim=(4, 1, 1), block_dim=(256, 1, 1))
    k.splitk_linear_layer(input=mid, weight=k.attach_input(torch.zeros(256, 1024, dtype=torch.bfloat16), "w2"), output=ws,
                          grid_dim=(2, 2, 1), block_dim=(256, 1, 1))
    k.splitk_reduce_layer(workspace=ws, residual=o1, output=o2, k_splits=2, grid_dim=(2, 1, 1), block_dim=(256, 1, 1))
    plan = k.plan().strip().splitlines()
    assert [ln.split()[1] for ln in plan] == ["linear", "silu_mul", "linear", "linear"]  # mid has a second reader: no fusion
    assert "split-k workspace + reduce folded" in plan[3] and "out=o2" in plan[3]
    k.finalize()
    k = _kernel(R=4, pages=16)
    with pytest.raises(NotImplementedError, match="splitk_reduce"):
        k.splitk_reduce_layer(workspace=k.new_tensor(dims=(8, 64), name="ws"), residual=k.new_tensor(dims=(4, 64), name="r"),
                              output=k.new_tensor(dims=(4, 64), name="o"), k_splits=2, grid_dim=(1, 1, 1), block_dim=(256, 1, 1))
        k.plan()
    k.finalize()


def test_attention_layer_needs_one_page_per_request(native_lib):
    k = _kernel(R=2, max_seq=64, page=64, pages=2)
    kc = k.attach_input(torch.zeros(2, 64, 2, 128, dtype=torch.bfloat16), "kc")
    vc = k.attach_input(torch.zeros(2, 64, 2, 128, dtype=torch.bfloat16), "vc")
    qn, kn = k.attach_input(torch.ones(128, dtype=torch.bfloat16), "qn"), k.attach_input(torch.ones(128, dtype=torch.bfloat16), "kn")
    cs = k.attach_input(torch.zeros(64, 128, dtype=torch.bfloat16), "cos")
    sn = k.attach_input(torch.zeros(64, 128, dtype=torch.bfloat16), "sin")
    qkv = k.new_tensor(dims=(2, 8 * 128), name="qkv")
    out = k.new_tensor(dims=(2, 4 * 128), name="out")
    k.attention_layer(input=qkv, k_cache=kc, v_cache=vc, q_norm=qn, k_norm=kn, cos_pos_embed=cs, sin_pos_embed=sn,
                      output=out, grid_dim=(2, 2, 1), block_dim=(128, 1, 1))
    assert k.plan().split()[1] == "attention"
    k.finalize()
    k = _kernel(R=2, max_seq=64, page=16, pages=8)
    kc = k.attach_input(torch.zeros(8, 16, 2, 128, dtype=torch.bfloat16), "kc")
    with pytest.raises(NotImplementedError, match="one page per request"):
        k.attention_layer(input=k.new_tensor(dims=(2, 1024), name="qkv"), k_cache=kc, v_cache=kc, q_norm=qn, k_norm=kn,
                          cos_pos_embed=cs, sin_pos_embed=sn, output=k.new_tensor(dims=(2, 512), name="o"),
                          grid_dim=(2, 2, 1), block_dim=(128, 1, 1))
    k.finalize()


def test_mpk_wrapper_builds_the_same_program(native_lib):
    """MPK fills in missing meta tensors and records the Qwen3 graph from checkpoint-named weights."""
    geom = mk.Qwen3Geometry(hidden=512, n_q=4, n_kv=2, mlp=1024, layers=2, vocab=2048)
    w = _weights(geom, 2)
    names = {"q": "self_attn.q_proj.weight", "k": "self_attn.k_proj.weight", "v": "self_attn.v_proj.weight",
             "o": "self_attn.o_proj.weight", "qn": "self_attn.q_norm.weight", "kn": "self_attn.k_norm.weight",
             "gate": "mlp.gate_proj.weight", "up": "mlp.up_proj.weight", "down": "mlp.down_proj.weight",
             "ln1": "input_layernorm.weight", "ln2": "post_attention_layernorm.weight"}
    sd = {"model.embed_tokens.weight": w["embed"], "model.norm.weight": w["norm"], "lm_head.weight": w["lm_head"]}
    for i in range(2):
        for s, l in names.items():
            sd[f"model.layers.{i}.{l}"] = w[f"l{i}.{s}"]
    kc = [torch.zeros(8, 16, 2, 128, dtype=torch.bfloat16) for _ in range(2)]
    cos = torch.zeros(64, 128, dtype=torch.bfloat16)
    mc = mk.MirageModelConfig(hidden_size=512, intermediate_size=1024, vocab_size=2048, local_num_q_heads=4,
                              local_num_kv_heads=2, head_dim=128, num_layers=2, k_cache=kc, v_cache=[t.clone() for t in kc],
                              position_embeddings=(cos, cos.clone()), state_dict=sd)
    meta = mk.MPKMetadata(mode="offline", total_num_requests=2, max_seq_length=64, max_num_batched_requests=2,
                          max_num_batched_tokens=2, max_num_pages=8, page_size=16, device="cpu", model_config=mc)
    m = mk.MPK(meta)
    assert m.tokens.shape == (2, 64) and m.qo_indptr_buffer.shape == (3,)
    m.build()
    kinds = [ln.split()[1] for ln in m.persistent_kernel.plan().strip().splitlines()]
    assert kinds == ["embed"] + ["linear", "attention", "linear", "linear", "linear"] * 2 + ["linear", "argmax_reduce"]
    with pytest.raises(NotImplementedError):
        m.load_new_request("a string prompt needs a tokenizer")
    m.load_new_request([5, 6, 7])
    assert m.tokens[1, :4].tolist() == [5, 6, 7, 0] and m.prompt_lengths.tolist() == [3, 3]
    m.finalize()


@pytest.mark.parametrize("tokens,depth", [(3, 4), (16, 4), (17, 3), (32, 3), (33, 3), (64, 3), (65, 2), (128, 2)])
def test_wide_ring_leaves_the_l1_its_share(native_lib, tokens, depth):
    """The ring beside the attention's scratch, as the product builds it: as many stages as stay within the 164 KB carve-out (with
    the 1 KB that the system adds): what the ring does not take is L1.  12 layers of 8B width, us per step: a stage more brings
    nothing up to 16 token rows (8 requests with 4, 5 and 6 stages 1249, 1270, 1269) and would be faster beyond (32 requests with 3
    and 4 1422, 1394; 64 1682, 1671; 100 with 2 and 3 2215, 2137, which need 210 KB); this is the depth that is built."""
    smem = C.c_int(0)
    attention = 8192 + 8 * 8 * 8  # the attention scratch: 8 KB to combine the warps' sums, (max, sum) pairs
    attention = (attention + 1023) // 1024 * 1024
    stages = native_lib.mk_debug_wide_ring(tokens, attention, C.byref(smem))
    assert stages == depth and smem.value + 1024 <= 164 * 1024
    stages = native_lib.mk_debug_wide_ring(tokens, 64 * 1024, C.byref(smem))  # (a norm of 32768 columns)
    assert stages >= 2 and smem.value <= 227 * 1024


@pytest.mark.parametrize("tokens", [1, 2, 3, 16, 17, 32, 33, 64, 65, 128])
def test_page_tables_are_rewritten_through_shared_memory(native_lib, tokens):
    """64 requests of 8192 tokens on 16-position pages are 32768 page numbers; deeper or shallower rings leave room for as many."""
    assert native_lib.mk_debug_page_entries(tokens, 8192 + 8 * 8 * 8) >= 32768


@pytest.mark.parametrize("widths,barrier", [((512, 512), True), ((512, 1024), False)])
def test_norm_rows_are_not_overwritten_while_the_linear_before_reads_them(widths, barrier):
    """Two fused norm linears with an allreduce between them, on the wide path: each norm becomes an op that stores its rows,
    into the same rows where the widths are equal.  The second takes its input word by word, without a barrier, but the
    linear before it may still be reading the first one's rows."""
    T, (k0, k1) = 4, widths
    k = mk.PersistentKernel(mode="online_notoken", world_size=2, mpi_rank=0, num_workers=0, num_local_schedulers=0, num_remote_schedulers=0,
                            max_seq_length=64, max_num_batched_requests=T, max_num_batched_tokens=T, max_num_pages=8, page_size=16,
                            meta_tensors=_meta(T, T, 64, 8), profiler_tensor=None, trace_name="", spec_decode_config=None, use_cutlass_kernel=True)
    held = []

    def attach(name, *shape):
        held.append(torch.zeros(shape, dtype=torch.bfloat16))
        return k.attach_input(held[-1], name)

    part, buf, red = k.new_tensor(dims=(T, k1), name="part"), k.new_tensor(dims=(2, T, k1), name="buf"), k.new_tensor(dims=(T, k1), name="red")
    k.rmsnorm_linear_layer(input=attach("x", T, k0), weight_norm=attach("n0", k0), weight_linear=attach("w0", k1, k0), output=part,
                           grid_dim=(8, 1, 1), block_dim=(128, 1, 1))
    k.allreduce_layer(input=part, buffer=buf, output=red, grid_dim=(8, 1, 1), block_dim=(128, 1, 1))
    k.rmsnorm_linear_layer(input=red, weight_norm=attach("n1", k1), weight_linear=attach("w1", 256, k1), output=attach("y", T, 256),
                           grid_dim=(4, 1, 1), block_dim=(128, 1, 1))
    buf_ = C.create_string_buffer(1 << 16)
    assert k._lib.mk_debug_describe_wide(k._h, buf_, 1 << 16) == 4
    ops = buf_.value.decode().strip().splitlines()
    assert [ln.split()[1] for ln in ops] == ["rmsnorm", "linear", "rmsnorm", "linear"]
    sync = [int(ln.split("flags=")[1].split()[0], 16) & 1 for ln in ops]
    assert sync == [0, 1, 1 if barrier else 0, 1], ops


@pytest.mark.parametrize("tokens,numerics,form,folded", [
    (3, "torch", "plain", True), (32, "torch", "plain", True), (33, "torch", "plain", False), (8, "mpk", "plain", True), (9, "mpk", "plain", False),
    (4, "torch", "user input", False), (4, "torch", "user output", False), (4, "torch", "second reader", False), (4, "torch", "in place", False),
    (4, "torch", "no linear before", False), (4, "torch", "residual of the rows", True)])
def test_norms_folded_into_activation_boxes(tokens, numerics, form, folded):
    """linear -> RMSNorm -> linear on the wide path: the norm goes into the second linear's boxes only where nobody else can see
    the normalised rows and the rows that are read meanwhile are the runtime's own."""
    n = 256
    k = mk.PersistentKernel(mode="online_notoken", world_size=1, mpi_rank=0, num_workers=0, num_local_schedulers=0, num_remote_schedulers=0,
                            max_seq_length=64, max_num_batched_requests=tokens, max_num_batched_tokens=tokens, max_num_pages=tokens, page_size=64,
                            meta_tensors=_meta(tokens, tokens, 64, tokens), profiler_tensor=None, trace_name="", spec_decode_config=None,
                            use_cutlass_kernel=True, numerics=numerics)
    held = []

    def attach(name, *shape):
        held.append(torch.zeros(shape, dtype=torch.bfloat16))
        return k.attach_input(held[-1], name)

    def own(name):
        return k.new_tensor(dims=(tokens, n), name=name)

    grid = dict(grid_dim=(4, 1, 1), block_dim=(128, 1, 1))
    h = attach("h", tokens, n) if form == "user input" else own("h")
    a = attach("a", tokens, n) if form == "user output" else own("a")
    y = h if form == "in place" else attach("y", tokens, n)
    if form == "no linear before":
        k.rmsnorm_layer(input=attach("x", tokens, n), weight=attach("n0", n), output=h, **grid)
    else:
        k.linear_layer(input=attach("x", tokens, n), weight=attach("w0", n, n), output=h, **grid)
    k.rmsnorm_layer(input=h, weight=attach("n1", n), output=a, **grid)
    if form == "residual of the rows":
        k.linear_with_residual_layer(input=a, weight=attach("w1", n, n), residual=h, output=y, **grid)
    else:
        k.linear_layer(input=a, weight=attach("w1", n, n), output=y, **grid)
    if form == "second reader":
        k.linear_layer(input=a, weight=attach("w2", n, n), output=attach("z", tokens, n), **grid)
    text = C.create_string_buffer(1 << 16)
    ops = k._lib.mk_debug_describe_wide(k._h, text, 1 << 16)
    assert ops == (4 if form == "second reader" else 3) - int(folded), text.value.decode()
    assert ("rmsnorm in the activation boxes" in text.value.decode()) == folded
    k.finalize()


def test_tagged_words_move_as_64_bit_scalars():
    """A word that carries the awaited number carries its value: the two halves travel in one 64-bit scalar, which is single-copy
    atomic.  The elements of a vector of 32-bit scalars may be of different ages."""
    csrc = os.path.join(os.path.dirname(mk.__file__), "csrc")
    found = set()
    for name in ("mk_kernel.cu", "mk_wide.cuh"):
        with open(os.path.join(csrc, name)) as f:
            found |= set(re.findall(r"(?:ld|st)\.relaxed\.(?:gpu|sys)\.global\.[\w.]+", f.read()))
    assert found and all(re.fullmatch(r"(ld|st)\.relaxed\.(gpu|sys)\.global\.(v2\.)?b64", form) for form in found), found
