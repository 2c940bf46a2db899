"""Whole-path parity on a B200: offline-mode greedy decode through the
PersistentKernel mirror against (a) the fixtures produced by the unmodified
reference PyTorch model and (b) the oracle run on the host on the same seeded
weights.  Tolerance (the stated one): per-step logits within 2e-2 of the step's
largest |logit| after bf16 rounding; greedy tokens identical.

Token equality needs care with random weights: bf16 logits tie or nearly tie
often (top-2 gap below one bf16 ulp), where any reordering of an fp32 sum flips
the argmax.  The tests therefore teacher-force the reference's tokens, require
the token to be identical at every step whose reference top-2 gap exceeds the
logit tolerance, and require it to be one of the reference's near-top
candidates elsewhere; the free-running identical prefix is checked on top."""
import os

import pytest
import torch

import fleet_chiplet_megakernel_b200 as mk
from oracle import qwen3_oracle as O
from tests.helpers import bf16_close, onepass_kernel

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
TOL = 2e-2


def _geom(g):
    return mk.Qwen3Geometry(hidden=g.hidden, n_q=g.n_q, n_kv=g.n_kv, head_dim=g.head_dim, mlp=g.mlp, layers=g.layers,
                            vocab=g.vocab, rope_theta=g.rope_theta)


def _cuda(w):
    return {k: v.cuda() for k, v in w.items()}


def _free_run(geom, w, prompts, n_new, numerics="torch", fuse=True, page_size=16, max_requests=None, num_layers=None):
    P = max(len(p) for p in prompts)
    dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=P + n_new, max_requests=max_requests or len(prompts),
                          total_requests=len(prompts), page_size=page_size, numerics=numerics, fuse=fuse,
                          num_layers=num_layers)
    dec.set_prompts(prompts)
    dec.run()
    out = [dec.generated(r).cpu().tolist() for r in range(len(prompts))]
    timing = dec.mpk.get_event_timing()
    dec.finalize()
    return out, timing


def _teacher_forced(geom, w, prompt, ref_tokens, n_new, numerics="torch", fuse=True, page_size=16, num_layers=None,
                    debug_flags=0):
    """One launch per iteration; after each, the reference's token replaces ours.
    Returns our per-step logits [n_new, vocab] and our greedy tokens."""
    P = len(prompt)
    dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=P + n_new + 1, max_requests=1, page_size=page_size,
                          numerics=numerics, fuse=fuse, keep_logits=True, max_iterations=1, num_layers=num_layers,
                          debug_flags=debug_flags)
    dec.set_prompts([prompt])
    logits, toks = [], []
    for it in range(P + n_new - 1):
        dec.run()
        if it >= P - 1:
            j = it - (P - 1)
            logits.append(dec.logits[0].clone().cpu())
            toks.append(int(dec.tokens[0, P + j]))
            dec.tokens[0, P + j] = int(ref_tokens[P + j])
    dec.finalize()
    return torch.stack(logits), toks


def _check_against(logits, toks, ref_logits, ref_tokens, P, what, TOL=TOL):
    n = logits.shape[0]
    err = O.max_rel_err(logits, ref_logits[:n])
    assert err <= TOL, f"{what}: logits off by {err:.4g} of the step's largest |logit|"
    scale = ref_logits[:n].float().abs().amax(-1)
    margin = O.top2_margin(ref_logits[:n])
    firm = 0
    for j in range(n):
        ref_tok = int(ref_logits[j].float().argmax())  # == the reference's greedy token
        if margin[j] > TOL * scale[j]:
            firm += 1
            assert toks[j] == ref_tok, f"{what}: step {j} token {toks[j]} != {ref_tok} (margin {float(margin[j]):.3g})"
        else:
            near = ref_logits[j].float()
            assert near[toks[j]] >= near.max() - TOL * scale[j], f"{what}: step {j} token is not a near-top candidate"
    return err, firm


@pytest.mark.parametrize("name", ["tiny_generate.pt", "small_generate.pt"])
@pytest.mark.parametrize("numerics,fuse", [("torch", True), ("torch", False), ("mpk", True)])
def test_generate_matches_reference_fixture(name, numerics, fuse):
    fx = torch.load(os.path.join(GOLD, name))
    geom = O.Geometry(**fx["geometry"])
    w = O.make_weights(geom, fx["seed"], norm_jitter=fx["norm_jitter"])
    P, n_new = len(fx["prompt"]), 33
    logits, toks = _teacher_forced(geom, w, fx["prompt"], fx["tokens"], n_new, numerics=numerics, fuse=fuse)
    ref_logits = fx["logits"]
    if numerics == "mpk":
        # the reference megakernel's task arithmetic (fp32 norms with eps) is its own reference:
        # teacher-force the same tokens through the oracle's restatement of it
        m = O.MpkRefModel(geom, w, fx["max_seq"])
        ref = fx["tokens"].tolist()
        rows = [m.step(ref[p], p) for p in range(P + n_new - 1)]
        ref_logits = torch.stack(rows[P - 1:])
    err, firm = _check_against(logits, toks, ref_logits, fx["tokens"], P, f"{name}/{numerics}/fuse={fuse}")
    print(f"{name} {numerics} fuse={fuse}: max logit error {err:.4g}, {firm}/{n_new} steps with a firm margin")


def test_free_running_prefix_matches_fixture():
    fx = torch.load(os.path.join(GOLD, "small_generate.pt"))
    geom = O.Geometry(**fx["geometry"])
    w = O.make_weights(geom, fx["seed"], norm_jitter=fx["norm_jitter"])
    P = len(fx["prompt"])
    out, timing = _free_run(geom, w, [fx["prompt"]], 40)
    ref = fx["tokens"].tolist()
    assert out[0][:P] == ref[:P]
    same = next((i for i, (a, b) in enumerate(zip(out[0], ref)) if a != b), len(ref))
    margin = O.top2_margin(fx["logits"])
    scale = fx["logits"].float().abs().amax(-1)
    print(f"free-running identical prefix: {same - P} generated tokens")
    if same < len(ref):
        j = same - P  # the first divergence must sit on a near tie of the reference
        assert margin[j] <= TOL * scale[j], f"diverged at step {j} with margin {float(margin[j]):.3g}"
    assert len(out[0]) == P + 40
    assert timing.shape[0] == P + 40 - 1 + 1  # iterations + the closing stamp


def test_continuous_batching_more_requests_than_slots():
    """5 requests with ragged prompts through 2 slots: every request's tokens equal
    what it generates alone (decode is batch-invariant; pages are recycled)."""
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    prompts = [O.make_prompt(geom, n, r) for r, n in enumerate([5, 9, 3, 12, 7])]
    max_seq = 12 + 10
    dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=max_seq, max_requests=2, total_requests=5, page_size=8,
                          max_num_pages=6)
    dec.set_prompts(prompts)
    dec.run()
    batched = [dec.tokens[r].cpu().tolist() for r in range(5)]
    steps = dec.step.cpu().tolist()
    dec.finalize()
    assert steps == [max_seq - 1] * 5
    for r, p in enumerate(prompts):
        solo, _ = _free_run(geom, w, [p], max_seq - len(p), page_size=8)
        assert solo[0] == batched[r], f"request {r} differs between batched and solo runs"


def test_identical_requests_give_identical_rows():
    """The reference driver's own self-check (demo.py:1281-1301)."""
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    p = O.make_prompt(geom, 6, 0)
    for B in (2, 4, 7):
        out, _ = _free_run(geom, w, [p] * B, 20)
        assert all(o == out[0] for o in out), f"batch {B}"


def test_wide_batch_requests_match_solo_runs():
    """12 and 40 ragged requests at once (activation boxes of 16 and 64 rows): every request's
    tokens equal its solo run up to the first near-tie of its own logits, and the step where they
    part is shown to be such a near-tie."""
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    for B in (12, 40):
        prompts = [O.make_prompt(geom, 3 + (r % 7), r) for r in range(B)]
        max_seq = 9 + 12
        dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=max_seq, max_requests=B, page_size=8)
        dec.set_prompts(prompts)
        dec.run()
        batched = [dec.tokens[r].cpu().tolist() for r in range(B)]
        dec.finalize()
        for r in (0, 5, B - 1):
            solo, _ = _free_run(geom, w, [prompts[r]], max_seq - len(prompts[r]), page_size=8)
            P = len(prompts[r])
            n = next((i for i, (a, b) in enumerate(zip(solo[0], batched[r])) if a != b), max_seq)
            assert n >= P, f"batch {B}: request {r} lost its prompt"
            if n >= max_seq:
                continue
            # The two paths add up in different orders, so a near-tie of the logits may flip: where the
            # runs part, both tokens must be within the logit tolerance of each other in the solo path.
            lg, _ = _teacher_forced(geom, w, prompts[r], batched[r], n - P + 1, page_size=8)
            row = lg[n - P].float()
            gap = abs(float(row[solo[0][n]]) - float(row[batched[r][n]]))
            assert gap <= TOL * float(row.abs().max()), \
                f"batch {B}: request {r} diverges from its solo run at position {n} without a near-tie (gap {gap:.4g})"
        # identical requests in one wide batch give identical rows
        out, _ = _free_run(geom, w, [prompts[0]] * B, 10, page_size=8)
        assert all(o == out[0] for o in out), f"batch {B}: identical requests differ"


def test_eos_retires_a_request():
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    p = O.make_prompt(geom, 6, 0)
    full, _ = _free_run(geom, w, [p], 12)
    eos = full[0][6 + 4]
    dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=6 + 12, max_requests=1, page_size=16, eos_token_id=eos)
    dec.set_prompts([p])
    dec.run()
    got = dec.generated(0).cpu().tolist()
    dec.finalize()
    first = full[0].index(eos, 6)
    assert got == full[0][: first + 1]


def test_single_layer_config_against_reference_fixture():
    """Config 1: one Qwen3-8B-geometry decoder layer, one decode step at position 1024."""
    from tests.golden.make_golden import config1_inputs
    fx = torch.load(os.path.join(GOLD, "config1_layer.pt"))
    w, hidden, kc, vc, L = config1_inputs()
    geom = O.Geometry(layers=1, vocab=8)
    for numerics in ("torch", "mpk"):
        k, meta, (indptr, indices) = onepass_kernel(1, max_seq=L + 8, page_size=64, seq_lens=[L + 1], numerics=numerics)
        kcache = torch.zeros(1, k.max_num_pages, 64, geom.n_kv, 128, dtype=torch.bfloat16)
        vcache = torch.zeros_like(kcache)
        for i, pg in enumerate(indices):
            n = min(64, L - i * 64)
            if n > 0:
                kcache[0, pg, :n] = kc[i * 64:i * 64 + n]
                vcache[0, pg, :n] = vc[i * 64:i * 64 + n]
        kcd, vcd = kcache.cuda(), vcache.cuda()
        cos, sin = mk.qwen3_graph.rope_tables(_geom(geom), L + 8, "cuda")
        wd = _cuda(w)
        x_in = hidden[None, :].cuda()
        # feed the hidden state in place of the embedding: a 1-row "embedding table" and token id 0
        wd["embed"] = x_in
        meta["input_tokens"].zero_()
        out_t = mk.build_qwen3_graph(k, _geom(geom), wd, kcd, vcd, cos, sin, meta["input_tokens"],
                                     meta["output_tokens"], num_layers=1, lm_head=False)
        k.compile()
        k()
        out = k.read_tensor(out_t)
        err = bf16_close(out[0], fx["out_hidden"], TOL, f"config 1 layer output ({numerics})")
        pg, slot = indices[L // 64], L % 64
        bf16_close(kcd[0, pg, slot].reshape(-1), fx["new_k"].reshape(-1), TOL, "appended K")
        bf16_close(vcd[0, pg, slot].reshape(-1), fx["new_v"].reshape(-1), TOL, "appended V")
        print(f"config 1 ({numerics}): max error {err:.4g} of the largest |hidden|")
        k.finalize()


def test_full_geometry_layers_against_host_oracle():
    """Qwen3-8B geometry at full width and vocabulary, 2 layers (the 36-layer run
    is the benchmark's): teacher-forced logits and tokens against the oracle run
    on the host cores with the same seeded weights."""
    geom = O.Geometry(layers=2)
    w = O.make_weights(geom, 0)
    prompt = O.make_prompt(geom, 8, 0)
    n_new = 8
    ref = O.TorchRefModel(geom, w, 32)
    ref_tokens, ref_logits = ref.generate(prompt, n_new)
    logits, toks = _teacher_forced(geom, w, prompt, torch.tensor(ref_tokens), n_new, page_size=64)
    err, firm = _check_against(logits, toks, ref_logits, torch.tensor(ref_tokens), len(prompt), "8B geometry, 2 layers")
    print(f"8B geometry x2 layers: max logit error {err:.4g}, {firm}/{n_new} firm steps")


def _teacher_forced_batch(geom, w_cuda, prompts, ref_tokens, iters, page_size=64, num_layers=None, **kw):
    """Ragged requests in one batch, one launch per iteration, the reference's tokens forced after
    each.  Returns per request the logits of its decode steps [n_r, vocab] and its greedy tokens."""
    B = len(prompts)
    maxP = max(len(p) for p in prompts)
    dec = mk.Qwen3Decoder(_geom(geom), w_cuda, max_seq_length=maxP + iters + 2, max_requests=B, page_size=page_size,
                          keep_logits=True, max_iterations=1, num_layers=num_layers, max_tokens_per_request=1, **kw)
    dec.set_prompts(prompts)
    logits = [[] for _ in range(B)]
    toks = [[] for _ in range(B)]
    for it in range(iters):
        dec.run()
        lg = dec.logits.clone().cpu()
        for r, p in enumerate(prompts):
            P = len(p)
            if it >= P - 1:
                j = it - (P - 1)
                logits[r].append(lg[r])
                toks[r].append(int(dec.tokens[r, P + j]))
                dec.tokens[r, P + j] = int(ref_tokens[r][P + j])
    dec.finalize()
    return [torch.stack(x) for x in logits], toks


def test_full_depth_model_32_decode_steps_against_host_oracle():
    """The benchmarked model itself: Qwen3-8B geometry, all 36 layers, full vocabulary, batch 1,
    8 prompt tokens + 32 teacher-forced decode steps against the oracle on the host cores.  The
    seeded weights are drawn on the GPU and copied to the host, so both sides hold the same bytes.

    At this depth bf16 activations amplify any difference in summation order: two executions of the
    reference model ITSELF drift apart by more than the 2e-2 that holds for a few layers.  The test
    measures that drift in place (the same torch ops of the reference model run on the host cores and
    through torch's GPU libraries, same weights, same forced tokens) and holds the megakernel to it:
    it may not be further from the host oracle than the reference's own GPU execution is (plus a
    quarter), and where the oracle's top-2 margin exceeds that drift the greedy token must be identical.
    The per-layer arithmetic itself is held to 2e-2 by the 2-layer case above and the per-op tests."""
    geom = O.QWEN3_8B
    wd = O.make_weights(geom, 0, device="cuda")
    w = {k: v.cpu() for k, v in wd.items()}
    prompt = O.make_prompt(geom, 8, 0)
    n_new = 32
    ref = O.TorchRefModel(geom, w, 48)
    ref_tokens, ref_logits = ref.generate(prompt, n_new)
    del ref
    second = O.TorchRefModel(geom, wd, 48, device="cuda")
    _, gpu_logits = second.generate(prompt, n_new, forced=ref_tokens[len(prompt):])
    del second
    drift = O.max_rel_err(gpu_logits, ref_logits)
    P = len(prompt)
    dec = mk.Qwen3Decoder(_geom(geom), wd, max_seq_length=P + n_new + 1, max_requests=1, page_size=64, keep_logits=True,
                          max_iterations=1)
    dec.set_prompts([prompt])
    logits, toks = [], []
    for it in range(P + n_new - 1):
        dec.run()
        if it >= P - 1:
            j = it - (P - 1)
            logits.append(dec.logits[0].clone().cpu())
            toks.append(int(dec.tokens[0, P + j]))
            dec.tokens[0, P + j] = int(ref_tokens[P + j])
    dec.finalize()
    logits = torch.stack(logits)
    err_vs_gpu = O.max_rel_err(logits, gpu_logits)
    bound = max(TOL, 1.25 * drift)
    # logits within the bound; the identical token wherever the oracle's top-2 margin exceeds it, one of the
    # oracle's near-top candidates elsewhere
    err, firm = _check_against(logits, toks, ref_logits, torch.tensor(ref_tokens), P, "8B geometry, 36 layers", TOL=bound)
    same = sum(int(toks[j] == int(ref_tokens[P + j])) for j in range(n_new))
    print(f"8B geometry x36 layers: megakernel vs host oracle {err:.4g}, vs the reference ops on the GPU {err_vs_gpu:.4g}; "
          f"the reference's own host-vs-GPU drift {drift:.4g}; {firm}/{n_new} steps with a margin above the bound, "
          f"{same}/{n_new} greedy tokens identical to the oracle's")


@pytest.mark.parametrize("B", [5, 20])
def test_wide_batches_at_full_width_against_host_oracle(B):
    """Qwen3-8B width and vocabulary, 2 layers, a batch of ragged requests on the stream-K
    mma.sync path (B = 5) and on the tcgen05 path (B = 20): every request's teacher-forced logits
    and tokens against its own run of the oracle (decode is batch-invariant)."""
    geom = O.Geometry(layers=2)
    wd = O.make_weights(geom, 0, device="cuda")
    w = {k: v.cpu() for k, v in wd.items()}
    prompts = [O.make_prompt(geom, 3 + (r * 5) % 7, r) for r in range(B)]
    iters = 14
    refs = []
    for p in prompts:
        m = O.TorchRefModel(geom, w, 32)
        refs.append(m.generate(p, iters - (len(p) - 1)))
    logits, toks = _teacher_forced_batch(geom, wd, prompts, [torch.tensor(t) for t, _ in refs], iters)
    worst, firm = 0.0, 0
    for r, p in enumerate(prompts):
        ref_tokens, ref_logits = refs[r]
        e, f = _check_against(logits[r], toks[r], ref_logits, torch.tensor(ref_tokens), len(p), f"batch {B} request {r}")
        worst, firm = max(worst, e), firm + f
    print(f"8B width x2 layers, batch {B}: max logit error {worst:.4g}, {firm} firm token checks")


def test_barrier_counter_wraps_inside_a_launch():
    """The grid barrier's 32-bit counter is started just below its wrap: a 30-token generation crosses
    it a few barriers in and must give the same tokens as a run that starts at zero."""
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    p = O.make_prompt(geom, 6, 0)
    base, _ = _free_run(geom, w, [p], 24)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    epoch0 = 2**32 // sms - 2
    dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=6 + 24, max_requests=1, page_size=16,
                          test_barrier_epoch=epoch0, timeout_ms=2000)
    dec.set_prompts([p])
    dec.run()
    got = dec.generated(0).cpu().tolist()
    dec.finalize()
    assert got == base[0]


@pytest.mark.parametrize("cluster", [2, 4])
@pytest.mark.parametrize("B", [1, 20])
def test_cluster_first_grid_barrier_gives_the_same_tokens(cluster, B):
    """The hierarchical grid barrier (thread-block clusters meet in shared memory first) against the flat one."""
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    prompts = [O.make_prompt(geom, 4 + r % 5, r) for r in range(B)]
    base, _ = _free_run(geom, w, prompts, 16)
    dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=max(len(p) for p in prompts) + 16, max_requests=B,
                          page_size=16, cluster_size=cluster, timeout_ms=2000)
    dec.set_prompts(prompts)
    dec.run()
    got = [dec.generated(r).cpu().tolist() for r in range(B)]
    dec.finalize()
    assert got == base


# ---- chunked prefill: a request inside its prompt is fed a chunk of it per iteration --------------
def _teacher_forced_chunked(geom, w, prompt, ref_tokens, n_new, budget, page_size=16, numerics="torch"):
    """One request, a token budget of `budget` per iteration, one launch per iteration: the logits that
    produced each generated token and the token itself, the reference's token forced afterwards."""
    P = len(prompt)
    dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=P + n_new + 1, max_requests=1, page_size=page_size,
                          numerics=numerics, keep_logits=True, max_iterations=1, max_num_batched_tokens=budget)
    dec.set_prompts([prompt])
    logits, toks, launches = [], [], 0
    while len(logits) < n_new:
        dec.run()
        launches += 1
        st = int(dec.step[0])  # tokens of the request processed so far
        if st >= P:
            n_it = int(dec.qo_indptr[1])  # tokens the request had in this iteration: the last one's logits count
            logits.append(dec.logits[n_it - 1].clone().cpu())
            toks.append(int(dec.tokens[0, st]))
            dec.tokens[0, st] = int(ref_tokens[st])
        assert launches < P + n_new + 4
    dec.finalize()
    return torch.stack(logits), toks, launches


@pytest.mark.parametrize("name,budget", [("tiny_generate.pt", 64), ("small_generate.pt", 64), ("small_generate.pt", 5),
                                         ("kv8_generate.pt", 16)])
def test_chunked_prefill_matches_reference_fixture(name, budget):
    """The fixtures come from the reference model's own multi-token prefill (demo/qwen3/demo.py:1196-1212)."""
    fx = torch.load(os.path.join(GOLD, name))
    geom = O.Geometry(**fx["geometry"])
    w = O.make_weights(geom, fx["seed"], norm_jitter=fx["norm_jitter"])
    P, n_new = len(fx["prompt"]), 24
    logits, toks, launches = _teacher_forced_chunked(geom, w, fx["prompt"], fx["tokens"], n_new, budget)
    assert launches == -(-P // budget) + n_new - 1, "the prompt must take ceil(P / budget) iterations"
    err, firm = _check_against(logits, toks, fx["logits"], fx["tokens"], P, f"{name} chunked prefill, budget {budget}")
    print(f"{name} budget {budget}: max logit error {err:.4g}, {firm}/{n_new} firm steps, {launches} iterations")


@pytest.mark.parametrize("P", [1, 7, 64, 65])
def test_chunked_prefill_prompt_lengths_against_oracle(P):
    """Prompts of 1, 7, 64 and 65 tokens with a budget of 64 (the last one takes two prefill iterations)."""
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    prompt = O.make_prompt(geom, P, 3)
    n_new = 10
    ref = O.TorchRefModel(geom, w, P + n_new + 2)
    ref_tokens, ref_logits = ref.generate(prompt, n_new)
    logits, toks, launches = _teacher_forced_chunked(geom, w, prompt, torch.tensor(ref_tokens), n_new, 64, page_size=8)
    assert launches == -(-P // 64) + n_new - 1
    err, firm = _check_against(logits, toks, ref_logits, torch.tensor(ref_tokens), P, f"prompt of {P} tokens")
    print(f"prompt {P}: max logit error {err:.4g}, {firm}/{n_new} firm steps")


@pytest.mark.parametrize("n_q,n_kv", [(8, 1), (16, 2), (4, 1)])
def test_tagged_activations_give_the_bits_the_barriers_give(n_q, n_kv):
    """Batch 1 with a context long enough for several chunks per kv head, four and eight q heads per kv head (the
    latter is the Qwen3-30B-A3B attention shape: the chunk CTAs merge slices of 1024 output elements between
    them).  Tagged activations change how an op learns that its input is there, not what it computes: the logits
    must be bit-identical to a run in which every op keeps its grid barrier.  16/2 heads also against the host
    oracle (the 2e-2 floor of this comparison is 0.017-0.024 on these seeds whichever way the ops synchronise)."""
    geom = O.Geometry(hidden=1024, n_q=n_q, n_kv=n_kv, mlp=2048, layers=2, vocab=2048)
    w = O.make_weights(geom, 6)
    P, n_new = 70, 8
    prompt = O.make_prompt(geom, P, 6)
    ref = O.TorchRefModel(geom, w, P + n_new + 2)
    ref_tokens, ref_logits = ref.generate(prompt, n_new)
    tagged, toks = _teacher_forced(geom, w, prompt, torch.tensor(ref_tokens), n_new, page_size=16)
    barriers, _ = _teacher_forced(geom, w, prompt, torch.tensor(ref_tokens), n_new, page_size=16, debug_flags=16)
    assert torch.equal(tagged, barriers)
    if (n_q, n_kv) == (16, 2):
        err, firm = _check_against(tagged, toks, ref_logits, torch.tensor(ref_tokens), P, f"{n_q} q heads on {n_kv} kv heads")
        print(f"{n_q}/{n_kv} heads: max logit error {err:.4g}, {firm}/{n_new} firm steps")


def test_chunked_prefill_with_more_requests_than_slots():
    """7 requests with ragged prompts through 3 slots and a budget of 16 tokens per iteration (prompt chunks
    and decode tokens share iterations, pages are recycled): every request generates what it generates
    alone with one token per iteration, up to a near-tie of its own logits."""
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    lens = [5, 21, 3, 40, 7, 1, 18]
    prompts = [O.make_prompt(geom, n, r) for r, n in enumerate(lens)]
    max_seq = 40 + 12
    dec = mk.Qwen3Decoder(_geom(geom), _cuda(w), max_seq_length=max_seq, max_requests=3, total_requests=len(lens),
                          page_size=8, max_num_pages=24, max_num_batched_tokens=16)
    dec.set_prompts(prompts)
    dec.run()
    batched = [dec.tokens[r].cpu().tolist() for r in range(len(lens))]
    steps = dec.step.cpu().tolist()
    timing = dec.mpk.get_event_timing()
    dec.finalize()
    assert steps == [max_seq - 1] * len(lens)
    assert int(timing[:-1, 1].max()) > 3, "some iteration must have carried a prompt chunk"
    for r, p in enumerate(prompts):
        solo, _ = _free_run(geom, w, [p], max_seq - len(p), page_size=8)
        n = next((i for i, (a, b) in enumerate(zip(solo[0], batched[r])) if a != b), max_seq)
        assert n >= len(p), f"request {r} lost its prompt"
        if n < max_seq:
            lg, _ = _teacher_forced(geom, w, p, batched[r], n - len(p) + 1, page_size=8)
            row = lg[n - len(p)].float()
            gap = abs(float(row[solo[0][n]]) - float(row[batched[r][n]]))
            assert gap <= TOL * float(row.abs().max()), f"request {r} diverges at {n} without a near-tie (gap {gap:.4g})"


def test_mpk_wrapper_generates_what_the_decoder_generates():
    """MPK / MPKMetadata (the reference's serving-side wrapper, python/mirage/mpk/mpk.py): metadata + a model
    config with checkpoint-named weights, build, compile, run a prompt."""
    geom = O.TINY
    w = O.make_weights(geom, 0, norm_jitter=0.25)
    p = O.make_prompt(geom, 6, 0)
    base, _ = _free_run(geom, w, [p], 14)
    long_names = {"q": "self_attn.q_proj.weight", "k": "self_attn.k_proj.weight", "v": "self_attn.v_proj.weight",
                  "o": "self_attn.o_proj.weight", "qn": "self_attn.q_norm.weight", "kn": "self_attn.k_norm.weight",
                  "gate": "mlp.gate_proj.weight", "up": "mlp.up_proj.weight", "down": "mlp.down_proj.weight",
                  "ln1": "input_layernorm.weight", "ln2": "post_attention_layernorm.weight"}
    sd = {"model.embed_tokens.weight": w["embed"].cuda(), "model.norm.weight": w["norm"].cuda(),
          "lm_head.weight": w["lm_head"].cuda()}
    for i in range(geom.layers):
        for s, l in long_names.items():
            sd[f"model.layers.{i}.{l}"] = w[f"l{i}.{s}"].cuda()
    max_seq, page, pages = 20, 16, 2
    kc = [torch.zeros(pages, page, geom.n_kv, 128, dtype=torch.bfloat16, device="cuda") for _ in range(geom.layers)]
    vc = [torch.zeros_like(t) for t in kc]
    cos, sin = mk.qwen3_graph.rope_tables(_geom(geom), max_seq, "cuda")
    mc = mk.MirageModelConfig(hidden_size=geom.hidden, intermediate_size=geom.mlp, vocab_size=geom.vocab,
                              local_num_q_heads=geom.n_q, local_num_kv_heads=geom.n_kv, head_dim=128,
                              num_layers=geom.layers, k_cache=kc, v_cache=vc, position_embeddings=(cos, sin), state_dict=sd)
    meta = mk.MPKMetadata(mode="offline", total_num_requests=1, max_seq_length=max_seq, max_num_batched_requests=1,
                          max_num_batched_tokens=8, max_num_pages=pages, page_size=page, model_config=mc,
                          eos_token_id=0x7FFFFFFF)
    m = mk.MPK(meta)
    m.build()
    m.compile()
    out = m.run(p)
    m.finalize()
    assert out[0].cpu().tolist() == base[0]


@pytest.mark.parametrize("pool,budget", [(30000, 128), (30000, 64), (8100, 8), (30000, 1)])
def test_large_page_pools(pool, budget):
    """Pools whose page table does not fit into shared memory beside the ring, and tables in use that do not: one-position
    pages and up to 7600 of them, against 64-position pages (the same arithmetic, whatever the pages: bit for bit)."""
    geom, R = O.TINY, 1 if budget == 1 else 8
    w = _cuda(O.make_weights(geom, 0, norm_jitter=0.25))
    prompts = [O.make_prompt(geom, 940 - 3 * r if budget > 8 else 30, r) for r in range(R)]
    P = max(len(p) for p in prompts)
    n_new = 10 if budget > 8 else 960 - P
    got = []
    for page, pages in ((1, pool), (64, None)):
        dec = mk.Qwen3Decoder(_geom(geom), w, max_seq_length=P + n_new, max_requests=R, page_size=page, max_num_pages=pages,
                              max_num_batched_tokens=budget, numerics="mpk", keep_logits=True)
        dec.set_prompts(prompts)
        dec.run()
        got.append(([dec.generated(r).cpu() for r in range(R)], dec.logits[:R].cpu()))
        dec.finalize()
    assert all(torch.equal(a, b) for a, b in zip(got[0][0], got[1][0]))
    assert torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("requests,length,budget", [(64, 620, 128), (5, 8000, 64)])
def test_page_tables_wider_than_the_ring(requests, length, budget):
    """Tables in use that do not fit into shared memory where the weight ring was, either (some 39000 entries): rewritten through
    global memory, with the results of 64-position pages, bit for bit."""
    geom, n_new = O.TINY, 6
    w = _cuda(O.make_weights(geom, 0, norm_jitter=0.25))
    prompts = [O.make_prompt(geom, length - n_new, r) for r in range(requests)]
    got = []
    for page, pages in ((1, requests * length + 64), (64, None)):
        dec = mk.Qwen3Decoder(_geom(geom), w, max_seq_length=length, max_requests=requests, page_size=page, max_num_pages=pages,
                              max_num_batched_tokens=budget, numerics="mpk", keep_logits=True)
        dec.set_prompts(prompts)
        dec.run()
        got.append(([dec.generated(r).cpu() for r in range(requests)], dec.logits[:requests].cpu()))
        dec.finalize()
    assert all(torch.equal(a, b) for a, b in zip(got[0][0], got[1][0]))
    assert torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("requests,budget", [(1, 1), (2, 2), (5, 5), (24, 24), (40, 40), (100, 100), (1, 64), (3, 20)])
def test_a_generation_behind_one_that_was_given_up(requests, budget):
    """A token id out of range ends a launch in its fourth iteration (its first, where prompts come in chunks), with weights under
    way, in shared memory and in tensor memory; the handle generates as a new one does afterwards."""
    geom, n_new = O.TINY, 8
    w = _cuda(O.make_weights(geom, 0, norm_jitter=0.25))
    prompts = [O.make_prompt(geom, 6, r) for r in range(requests)]
    bad = [p.clone() for p in prompts]
    bad[-1][3] = geom.vocab
    got = []
    for spoil in (True, False):
        dec = mk.Qwen3Decoder(_geom(geom), w, max_seq_length=6 + n_new, max_requests=requests, page_size=16, max_num_batched_tokens=budget,
                              numerics="mpk", keep_logits=True)
        for _ in range(2 if spoil else 0):
            dec.set_prompts(bad)
            with pytest.raises(RuntimeError, match="token id out of range"):
                dec.run()
        dec.set_prompts(prompts)
        dec.run()
        got.append(([dec.generated(r).cpu() for r in range(requests)], dec.logits[:requests].cpu()))
        dec.finalize()
    assert all(torch.equal(a, b) for a, b in zip(got[0][0], got[1][0]))
    assert torch.equal(got[0][1], got[1][1])
