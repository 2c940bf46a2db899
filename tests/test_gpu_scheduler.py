"""The scheduler between two iterations (admission, prompt chunks under a token budget, pages, retirement), against the same rules
followed request by request on the host."""
import pytest
import torch

import fleet_chiplet_megakernel_b200 as mk
from oracle import qwen3_oracle as O

pytestmark = pytest.mark.gpu


class _Host:
    """One request after the other, as the reference's offline mode does it."""

    def __init__(self, lens, slots, budget, cap, page, pool, seq):
        self.lens, self.slots, self.budget, self.cap, self.page, self.pool, self.seq = lens, slots, budget, cap, page, pool, seq
        self.queue, self.head, self.tail = list(range(pool)), 0, pool
        self.waited = 0  # iterations in which a request waited for pages
        self.next, self.running = 0, []  # running: [request, step, tokens of the iteration, pages]

    def finish(self, tokens=None, eos=None):
        left = []
        for q in self.running:
            q[1] += q[2]
            ended = tokens is not None and q[1] >= self.lens[q[0]] and int(tokens[q[0], q[1]]) == eos
            if q[1] + 1 < self.seq and not ended:
                left.append(q)
            else:
                for pg in q[3]:
                    self.queue[self.tail % self.pool] = pg
                    self.tail += 1
        self.running = left

    def _pages(self, q):
        while len(q[3]) < -(-(q[1] + q[2]) // self.page):
            assert self.tail > self.head
            q[3].append(self.queue[self.head % self.pool])
            self.head += 1

    def prepare(self):
        used = 0
        for q in self.running:
            left = self.lens[q[0]] - q[1]
            q[2] = min(left, self.cap, self.budget - used) if left > 0 else min(1, self.budget - used)
            used += q[2]
            self._pages(q)
        while len(self.running) < self.slots and used < self.budget and self.next < len(self.lens):
            n = max(1, min(self.lens[self.next], self.cap, self.budget - used))
            if self.tail - self.head < -(-n // self.page):
                self.waited += 1
                break
            q = [self.next, 0, n, []]
            self._pages(q)
            self.running.append(q)
            self.next += 1
            used += n
        return used


def _decoder(slots, total, budget, cap, page, pool, seq, iterations, lens, eos=0x7FFFFFFF):
    geom = O.TINY
    g = mk.Qwen3Geometry(hidden=geom.hidden, n_q=geom.n_q, n_kv=geom.n_kv, mlp=geom.mlp, layers=1, vocab=geom.vocab)
    w = {k: v.cuda() for k, v in O.make_weights(geom, 0).items() if not k.startswith("l") or k.startswith(("l0.", "lm_head"))}
    gen = torch.Generator().manual_seed(total * slots)
    if lens is None:
        lens = torch.randint(1, seq - 3, (total,), generator=gen).tolist()
    prompts = [torch.randint(0, geom.vocab, (n,), generator=gen) for n in lens]
    dec = mk.Qwen3Decoder(g, w, max_seq_length=seq, max_requests=slots, total_requests=total, page_size=page, max_num_pages=pool,
                          max_num_batched_tokens=budget, max_tokens_per_request=cap, max_iterations=iterations, eos_token_id=eos)
    dec.set_prompts(prompts)
    return dec, prompts, _Host(lens, slots, max(slots, budget), cap or max(slots, budget), page, pool, seq)


def _as_prepared(dec, state, pages, slots, page):
    """The iteration that the decoder ran last, against what the host prepared."""
    n = len(state)
    qo = [0]
    kv = [0]
    for q, pg in zip(state, pages):
        qo.append(qo[-1] + q[2])
        kv.append(kv[-1] + len(pg))
    assert dec.qo_indptr.tolist() == qo + [qo[-1]] * (slots - n)
    assert dec.kv_indptr.tolist() == kv + [kv[-1]] * (slots - n)
    assert dec.kv_indices[:kv[-1]].tolist() == [p for pg in pages for p in pg]
    assert dec.kv_last_page_len[:n].tolist() == [(q[1] + q[2] - 1) % page + 1 for q in state]
    tokens, fed = dec.tokens.cpu(), dec.input_tokens[:, 0].cpu()
    for q, at in zip(state, qo):
        assert torch.equal(fed[at:at + q[2]], tokens[q[0], q[1]:q[1] + q[2]]), q


def _follow(dec, prompts, host, slots, page, iterations, eos=None):
    for _ in range(400):
        used = 0
        for _ in range(iterations):
            used = host.prepare()
            if used == 0:
                break
            want = [list(map(list, (q[:3] for q in host.running))), [list(q[3]) for q in host.running]]
            if eos is None:
                host.finish()
        dec.run()
        if used == 0:
            break
        _as_prepared(dec, *want, slots, page)
        if eos is not None:  # (an iteration at a time: what it generated decides who ends)
            host.finish(dec.tokens.cpu(), eos)
    assert used == 0
    for r, p in enumerate(prompts):
        assert torch.equal(dec.tokens[r, :len(p)].cpu(), p)


@pytest.mark.parametrize("slots,total,budget,cap,page,pool,seq,iterations", [
    (1, 3, 1, 0, 4, 8, 24, 5), (2, 7, 64, 0, 4, 20, 30, 3), (3, 3, 3, 0, 16, 9, 40, 4), (8, 24, 64, 0, 4, 80, 33, 7), (8, 20, 20, 9, 8, 40, 37, 4),
    (13, 40, 20, 0, 2, 200, 30, 6), (64, 64, 128, 0, 16, 200, 45, 5), (33, 90, 40, 1, 4, 264, 31, 9), (128, 300, 128, 16, 4, 1024, 29, 11)])
def test_every_iteration_is_prepared_as_one_request_after_the_other(slots, total, budget, cap, page, pool, seq, iterations):
    dec, prompts, host = _decoder(slots, total, budget, cap, page, pool, seq, iterations, None)
    _follow(dec, prompts, host, slots, page, iterations)
    assert dec.step.tolist() == [seq - 1] * total
    dec.finalize()


# Pools that hold fewer requests than there are places: some wait while others run, with places and budget to spare.  All of a
# request's pages are there when it is admitted (seq - 1 positions after a prompt of seq - 4 or more), so none runs out later.
@pytest.mark.parametrize("slots,total,budget,cap,page,pool,seq,iterations", [
    (2, 7, 64, 0, 4, 9, 24, 3), (8, 24, 64, 0, 4, 20, 24, 1), (8, 24, 128, 0, 4, 33, 24, 4), (33, 70, 128, 0, 2, 42, 17, 2), (128, 200, 128, 0, 16, 11, 16, 5)])
def test_requests_wait_for_pages(slots, total, budget, cap, page, pool, seq, iterations):
    gen = torch.Generator().manual_seed(pool)
    lens = torch.randint((seq - 2) // page * page + 1, seq - 1, (total,), generator=gen).tolist()
    dec, prompts, host = _decoder(slots, total, budget, cap, page, pool, seq, iterations, lens)
    _follow(dec, prompts, host, slots, page, iterations)
    assert host.waited > 0 and dec.step.tolist() == [seq - 1] * total
    dec.finalize()


@pytest.mark.parametrize("slots,total,budget,page,pool,seq", [(5, 17, 5, 4, 60, 40), (13, 40, 30, 4, 140, 40), (70, 130, 128, 8, 400, 40)])
def test_requests_that_end_early_make_room_in_the_middle_of_the_list(slots, total, budget, page, pool, seq):
    lens = [1 + (5 * r) % 11 for r in range(total)]
    dec, _, _ = _decoder(slots, total, budget, 0, page, pool, seq, 0, lens)
    dec.run()
    made = [dec.tokens[r, lens[r]:].tolist() for r in range(total)]
    dec.finalize()
    # the end token: the one that would end requests at the most different lengths
    eos = max({t for m in made for t in m}, key=lambda t: len({m.index(t) + n for m, n in zip(made, lens) if t in m}))
    dec, prompts, host = _decoder(slots, total, budget, 0, page, pool, seq, 1, lens, eos)
    _follow(dec, prompts, host, slots, page, 1, eos)
    # (the step of a request that has ended is the position of its last token)
    ends = [n + m.index(eos) if eos in m else seq - 1 for n, m in zip(lens, made)]
    assert len(set(ends)) > 2 and dec.step.tolist() == ends
    dec.finalize()


def test_a_pool_that_runs_dry_is_reported_and_nobody_is_lost():
    """Request 0 ends when the five others all need their second page: its two pages go to the first two, the third gets none.  A
    second launch finds the same: request 0 has ended and its pages are free."""
    slots, page, seq = 6, 4, 9
    dec, prompts, _ = _decoder(slots, slots, 10, 0, page, 7, seq, 0, [5, 1, 1, 1, 1, 1])
    for _ in range(2):
        with pytest.raises(RuntimeError, match=r"out of KV pages .* detail 3/2 "):
            dec.run()
        assert dec.step.tolist() == [seq - 1] + [4] * 5
    dec.set_prompts(prompts)  # (a new generation starts with all pages free)
    with pytest.raises(RuntimeError, match=r"out of KV pages .* detail 3/2 "):
        dec.run()
    dec.finalize()
