"""What a user of this framework has it do, as cases that can be timed and compared.

Three ways in:

* ``generate``: offline generation, ``Qwen3Decoder.set_prompts`` (host prompts) + ``run``: chunked prefill,
  then greedy decode steps until every sequence is ``seq`` tokens long; with more requests than slots the
  scheduler retires and admits requests on the way;
* ``step``: one pass of a ``PersistentKernel`` in mode ``online_notoken`` over metadata that the caller owns
  (page tables, last page lengths, input tokens), as a serving engine drives it token by token;
* ``moe``: the mixture-of-experts decoder (one or two requests, prompts advance one token per iteration).

Every pass returns what the path computes: tokens, request positions, the logits of the last iteration, and
the K/V caches with every row that was appended.

The weights are seeded, N(0, 0.02), with the projections into the residual stream scaled by
1/sqrt(2 layers) as in common initialisations; row next(t) of the LM head follows the embedding of t, so that
greedy decoding picks its tokens by a wide margin, as a trained model mostly does, and two correct
implementations generate the same tokens.
"""
import math

import torch

import fleet_chiplet_megakernel_b200 as mk

D = 128  # head dimension of the framework

# widths of the dense geometries: hidden, q heads, kv heads, MLP width, vocabulary
WIDTHS = {
    "tiny": (512, 4, 2, 1024, 2048),        # the test suite's smallest model
    "small": (1024, 8, 2, 3072, 8192),      # the test suite's small model
    "kv8": (1024, 16, 8, 3072, 8192),       # the test suite's model with eight kv heads
    "ragged": (1152, 8, 8, 2176, 32008),    # hidden width and vocabulary not multiples of the tiles
    "medium": (2048, 16, 8, 6144, 151936),
    "8b": (4096, 32, 8, 12288, 151936),     # the benchmark's geometry (36 layers)
}
# widths of the MoE geometries: hidden, q heads, kv heads, experts, top-k, expert MLP width, vocabulary
MOE_WIDTHS = {
    "moe_tiny": (512, 8, 2, 16, 4, 256, 2048),       # the test suite's
    "a3b": (2048, 32, 4, 128, 8, 768, 151936),       # the benchmark's (48 layers hold 60 GB: cut in depth here)
}


def listed():
    def gen(name, width, layers, batch, lo, hi, seq, **kw):
        c = {"name": name, "kind": "generate", "width": width, "layers": layers, "batch": batch, "total": batch,
             "prompt_lo": lo, "prompt_hi": hi, "seq": seq, "page": 64, "budget": 64, "numerics": "torch"}
        c.update(kw)
        return c

    return [
        # a small model answering with a few tokens: launches, host work and latency, hardly any bytes
        gen("small_model_b1", "small", 4, 1, 7, 7, 19, page=16),
        # one decoder layer at the benchmark's width, one token behind 1024 cached ones: the unit a serving
        # engine's integration test (and the benchmark's CPU leg) steps
        {"name": "layer_step_b1", "kind": "step", "width": "8b", "layers": 1, "batch": 1, "ctx_lo": 1024, "ctx_hi": 1024,
         "page": 64, "numerics": "torch"},
        # a serving engine's decode step over eight running requests of different ages
        {"name": "model_step_b8", "kind": "step", "width": "8b", "layers": 36, "batch": 8, "ctx_lo": 90, "ctx_hi": 1100,
         "page": 64, "numerics": "torch"},
        # the headline: one user, a 64-token prompt, 32 new tokens
        gen("chat_b1", "8b", 36, 1, 64, 64, 96),
        # one user with a long prompt and a short answer: prefill in 64-token chunks
        gen("long_prompt_b1", "8b", 36, 1, 1000, 1000, 1016),
        # two users (the widest batch of the small-batch path)
        gen("chat_b2", "8b", 36, 2, 40, 64, 88),
        # four users
        gen("chat_b4", "8b", 36, 4, 64, 64, 92),
        # thirteen requests of all lengths, the reference megakernel's roundings, shared prefill budget
        gen("ragged_b13", "8b", 36, 13, 17, 90, 98, numerics="mpk"),
        # continuous batching: 24 requests through 8 slots of a half-depth model
        gen("queue_24_over_8", "8b", 18, 8, 10, 40, 56, total=24),
        # throughput serving
        gen("batch_32", "8b", 36, 32, 64, 64, 80),
        gen("batch_64", "8b", 36, 64, 40, 40, 60, budget=128),
        # mixture of experts at the benchmark's widths
        {"name": "moe_b1", "kind": "moe", "width": "a3b", "layers": 12, "batch": 1, "prompt_lo": 16, "prompt_hi": 16, "seq": 40,
         "page": 64, "numerics": "mpk"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 200.0)


def draw(rng):
    limit = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["generate", "generate", "generate", "step", "step", "moe"])
        if kind == "moe":
            width = rng.choice(["moe_tiny", "a3b", "a3b"])
            lo = _log_int(rng, 1, 40)
            case = {"kind": kind, "width": width, "layers": rng.randint(2, 12 if width == "a3b" else 24), "batch": rng.choice([1, 1, 2]),
                    "prompt_lo": lo, "prompt_hi": lo + rng.randint(0, 9), "seq": lo + 9 + _log_int(rng, 4, 64)}
        else:
            width = rng.choice(["tiny", "small", "kv8", "ragged", "medium", "8b", "8b", "8b"])
            case = {"kind": kind, "width": width, "layers": _log_int(rng, 2, 36) if width in ("medium", "8b") else rng.randint(2, 12),
                    "batch": _log_int(rng, 1, 64)}
            if kind == "step":
                case["layers"] = rng.choice([1, case["layers"]])
                case["ctx_lo"] = _log_int(rng, 1, 600)
                case["ctx_hi"] = case["ctx_lo"] + _log_int(rng, 1, 600)
                most = case["ctx_hi"] + 1
            else:
                case["total"] = case["batch"] if rng.random() < 0.7 else case["batch"] + rng.randint(1, 2 * case["batch"] + 2)
                case["prompt_lo"] = _log_int(rng, 1, 700)
                case["prompt_hi"] = case["prompt_lo"] + rng.choice([0, _log_int(rng, 1, 300)])
                case["seq"] = most = case["prompt_hi"] + _log_int(rng, 4, 64)
                # the token budget of an iteration: one token per request, or room for prompt chunks
                case["budget"] = rng.choice([case["batch"], 64, 64, 128, max(case["batch"], rng.randint(3, 100))])
                case["budget"] = max(case["budget"], case["batch"])
            if case["batch"] * most > 16384:
                continue
        case["page"] = rng.choice([16, 64, 64])
        case["numerics"] = rng.choice(["torch", "torch", "mpk"])
        if _cost(case) <= limit:
            return case


# ------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------
def _geometry(case):
    if case["kind"] == "moe":
        h, nq, nkv, e, k, m, v = MOE_WIDTHS[case["width"]]
        return mk.Qwen3MoeGeometry(hidden=h, n_q=nq, n_kv=nkv, experts=e, top_k=k, moe_mlp=m, layers=case["layers"], vocab=v)
    h, nq, nkv, m, v = WIDTHS[case["width"]]
    return mk.Qwen3Geometry(hidden=h, n_q=nq, n_kv=nkv, mlp=m, layers=case["layers"], vocab=v)


def _weights(g, seed, moe):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)

    def rnd(*shape, std=0.02):
        return torch.randn(shape, generator=gen, dtype=torch.bfloat16, device=dev).mul_(std)

    def norm(n):
        return (1.0 + 0.25 * (2 * torch.rand(n, generator=gen, device=dev) - 1)).to(torch.bfloat16)

    into = 0.02 / math.sqrt(2 * g.layers)  # projections into the residual stream
    w = {"embed": rnd(g.vocab, g.hidden, std=1.0)}
    previous = torch.randperm(g.vocab, generator=gen, device=dev)
    w["lm_head"] = w["embed"][previous].mul_(0.02)
    for i in range(g.layers):
        w[f"l{i}.q"], w[f"l{i}.k"], w[f"l{i}.v"] = rnd(g.n_q * D, g.hidden), rnd(g.n_kv * D, g.hidden), rnd(g.n_kv * D, g.hidden)
        w[f"l{i}.o"] = rnd(g.hidden, g.n_q * D, std=into)
        if moe:
            w[f"l{i}.router"] = rnd(g.experts, g.hidden, std=2.0 / g.hidden ** 0.5)
            w[f"l{i}.w13"] = rnd(g.experts, 2 * g.moe_mlp, g.hidden)
            w[f"l{i}.w2"] = rnd(g.experts, g.hidden, g.moe_mlp, std=into)
        else:
            w[f"l{i}.gate"], w[f"l{i}.up"] = rnd(g.mlp, g.hidden), rnd(g.mlp, g.hidden)
            w[f"l{i}.down"] = rnd(g.hidden, g.mlp, std=into)
        w[f"l{i}.ln1"], w[f"l{i}.ln2"], w[f"l{i}.qn"], w[f"l{i}.kn"] = norm(g.hidden), norm(g.hidden), norm(D), norm(D)
    w["norm"] = norm(g.hidden)
    return w


def _spread(lo, hi, n):
    """n lengths over [lo, hi], in a mixed order (the same for every seed)."""
    if n == 1:
        return [hi]
    v = [lo + (hi - lo) * i // (n - 1) for i in range(n)]
    return [v[(i * 5) % n] for i in range(n)] if n % 5 else v[::-1]


class _Generate:
    def __init__(self, case, seed):
        g = _geometry(case)
        moe = case["kind"] == "moe"
        self.weights = _weights(g, seed, moe)
        lens = _spread(case["prompt_lo"], case["prompt_hi"], case.get("total", case["batch"]))
        gen = torch.Generator().manual_seed(seed)
        self.prompts = [torch.randint(0, g.vocab, (n,), generator=gen, dtype=torch.int64) for n in lens]
        kw = dict(max_seq_length=case["seq"], max_requests=case["batch"], total_requests=len(lens), page_size=case["page"],
                  numerics=case["numerics"], keep_logits=True)
        if moe:
            self.dec = mk.Qwen3MoeDecoder(g, self.weights, **kw)
        else:
            self.dec = mk.Qwen3Decoder(g, self.weights, max_num_batched_tokens=case["budget"], **kw)

    def run(self):
        d = self.dec
        d.set_prompts(self.prompts)
        d.run()
        return {"tokens": d.tokens, "step": d.step, "logits": d.logits, "k_cache": d.k_cache, "v_cache": d.v_cache}


class _Step:
    """The caller owns the paging metadata; requests sit on pages scattered over the pool."""

    def __init__(self, case, seed):
        g = _geometry(case)
        dev = torch.device("cuda")
        self.weights = _weights(g, seed, False)
        R, page = case["batch"], case["page"]
        lens = [n + 1 for n in _spread(case["ctx_lo"], case["ctx_hi"], R)]  # the new token included
        pages = [math.ceil(n / page) for n in lens]
        total = sum(pages)
        gen = torch.Generator().manual_seed(seed)
        indptr = torch.zeros(R + 1, dtype=torch.int32)
        indptr[1:] = torch.cumsum(torch.tensor(pages), 0)
        self.meta = {
            "step": torch.zeros(R, dtype=torch.int32, device=dev),
            "tokens": torch.zeros(R, max(lens) + 1, dtype=torch.int64, device=dev),
            "input_tokens": torch.randint(0, g.vocab, (R, 1), generator=gen, dtype=torch.int64).to(dev),
            "output_tokens": torch.zeros(R, 1, dtype=torch.int64, device=dev),
            "num_new_tokens": torch.ones(R, dtype=torch.int32, device=dev),
            "prompt_lengths": torch.ones(R, dtype=torch.int32, device=dev),
            "qo_indptr_buffer": torch.arange(R + 1, dtype=torch.int32, device=dev),
            "paged_kv_indptr_buffer": indptr.to(dev),
            "paged_kv_indices_buffer": torch.randperm(total, generator=gen).to(torch.int32).to(dev),
            "paged_kv_last_page_len_buffer": torch.tensor([n - (p - 1) * page for n, p in zip(lens, pages)], dtype=torch.int32, device=dev),
        }
        dgen = torch.Generator(device=dev).manual_seed(seed + 1)
        shape = (g.layers, total, page, g.n_kv, D)
        self.k_cache = torch.randn(shape, generator=dgen, dtype=torch.bfloat16, device=dev)
        self.v_cache = torch.randn(shape, generator=dgen, dtype=torch.bfloat16, device=dev)
        self.logits = torch.zeros(R, g.vocab, dtype=torch.bfloat16, device=dev)
        inv = 1.0 / (g.rope_theta ** (torch.arange(0, D, 2, dtype=torch.float32) / D))
        ang = torch.arange(max(lens) + 1, dtype=torch.float32)[:, None] * inv[None, :]
        ang = torch.cat((ang, ang), dim=-1)
        self.cos, self.sin = ang.cos().to(torch.bfloat16).to(dev), ang.sin().to(torch.bfloat16).to(dev)
        self.kernel = mk.PersistentKernel(
            mode="online_notoken", world_size=1, mpi_rank=0, num_workers=0, num_local_schedulers=0, num_remote_schedulers=0,
            max_seq_length=max(lens) + 1, max_num_batched_requests=R, max_num_batched_tokens=R, max_num_pages=total, page_size=page,
            meta_tensors=self.meta, numerics=case["numerics"])
        mk.build_qwen3_graph(self.kernel, g, self.weights, self.k_cache, self.v_cache, self.cos, self.sin, self.meta["input_tokens"],
                             self.meta["output_tokens"], logits=self.logits)
        self.kernel.compile()

    def run(self):
        self.kernel()
        return {"next": self.meta["output_tokens"], "logits": self.logits, "k_cache": self.k_cache, "v_cache": self.v_cache}


def prepare(case, seed):
    return _Step(case, seed) if case["kind"] == "step" else _Generate(case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------
def _iterations(case):
    """The schedule of a pass: per iteration a list of (first position, tokens) of the requests it serves."""
    if case["kind"] == "step":
        return [[(n, 1) for n in _spread(case["ctx_lo"], case["ctx_hi"], case["batch"])]]
    moe = case["kind"] == "moe"
    waiting = list(_spread(case["prompt_lo"], case["prompt_hi"], case.get("total", case["batch"])))
    budget, cap = (case["batch"], 1) if moe else (case["budget"], case["budget"])
    running, out = [], []
    while True:
        running = [r for r in running if r[0] + 1 < case["seq"]]
        served, left = [], budget
        for r in running:
            n = min(r[1] - r[0], cap, left) if r[1] > r[0] else min(1, left)
            if n > 0:
                served.append((r[0], n))
            r[0] += n
            left -= n
        while waiting and len(running) < case["batch"] and left > 0:
            p = waiting.pop(0)
            n = min(p, cap, left)
            served.append((0, n))
            running.append([n, p])
            left -= n
        if not served:
            return out
        out.append(served)


def work(case):
    g = _geometry(case)
    moe = case["kind"] == "moe"
    attn = g.hidden * (g.n_q + 2 * g.n_kv) * D + g.hidden * g.n_q * D
    head = g.vocab * g.hidden
    if moe:
        expert = 3 * g.moe_mlp * g.hidden
        router = g.experts * g.hidden
        per_token = g.layers * (attn + router + g.top_k * expert) + head
    else:
        per_token = g.layers * (attn + 3 * g.mlp * g.hidden) + head
    nbytes = flops = 0.0
    for served in _iterations(case):
        t = sum(n for _, n in served)
        if moe:
            # the experts that t tokens choose between them, were the choices independent
            used = g.experts * (1 - (1 - g.top_k / g.experts) ** t)
            nbytes += 2 * (g.layers * (attn + router + used * expert) + head)
        else:
            nbytes += 2 * per_token
        nbytes += t * (2 * g.vocab + 2 * g.hidden)                                    # logits written, embedding rows read
        nbytes += sum(4 * g.layers * g.n_kv * D * (p + 2 * n) for p, n in served)      # K/V rows read once, new ones written
        flops += 2.0 * per_token * t
        flops += sum(4.0 * g.layers * g.n_q * D * (p * n + n * (n + 1) / 2) for p, n in served)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # A layer passes values through two bf16 residual additions and some ten more bf16 roundings.  Another order of
    # summation flips some of them, and behind a few layers two correct runs round independently of one another:
    # about 1e-2 (2-norm) for one layer, growing like the square root of the depth.  Measured with the grid cut to 131
    # CTAs (another split of every sum): 0.003 behind 4 layers, 0.024 behind 36, largest single difference 0.19 of the
    # root mean square among tens of millions.  A MoE router may flip a near-tie besides.  Tokens are chosen by wide
    # margins: equal.
    return {"rel": 3e-2 if case["kind"] == "moe" else min(3e-2, 1e-2 * math.sqrt(case["layers"])), "max": 0.4}
