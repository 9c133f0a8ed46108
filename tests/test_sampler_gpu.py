"""Device sampler (csrc/sampler.cu) against the host policy ``sample_row``."""
import math

import pytest
import torch

from scirust_b200.generate import SamplerRng, SamplingParams, sample_row
from scirust_b200.models import GQADecoder, SciAgentConfig
from scirust_b200.models.infer import InferenceEngine
from scirust_b200.ops.sampling import DeviceSampler

pytestmark = pytest.mark.gpu


def _logits(rows, vocab, seed, scale=3.0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(rows, vocab, generator=g) * scale


def test_greedy_with_repetition_penalty_matches_host():
    rows, vocab = 6, 5000
    lg = _logits(rows, vocab, 1)
    params = SamplingParams(temperature=0.0, repetition_penalty=1.3, repetition_window=16)
    hist = torch.stack([lg[b].topk(20).indices for b in range(rows)])       # penalise the current leaders
    hist[:, 5] = hist[:, 4]                                                 # a repeated token is penalised twice
    s = DeviceSampler(params, rows, vocab, range(rows), "cuda", history_len=32)
    s.set_history(hist)
    got = s.sample(lg.cuda()).cpu()
    want = [sample_row(lg[b], params, hist[b].tolist(), SamplerRng(b)) for b in range(rows)]
    assert got.tolist() == want


def test_top_k_one_is_argmax_and_ties_take_the_lower_id():
    lg = _logits(4, 1000, 2)
    lg[0, 17] = lg[0, 900] = 50.0
    s = DeviceSampler(SamplingParams(temperature=0.8, top_k=1), 4, 1000, [3, 4, 5, 6], "cuda")
    got = s.sample(lg.cuda()).cpu().tolist()
    assert got[0] == 17
    assert got[1:] == lg[1:].argmax(-1).tolist()


@pytest.mark.parametrize("params", [SamplingParams(temperature=1.0), SamplingParams(temperature=0.7, top_k=50),
                                    SamplingParams(temperature=1.2, top_p=0.9),
                                    SamplingParams(temperature=0.9, top_k=200, top_p=0.8, repetition_penalty=1.2)])
def test_same_seed_same_token_as_host(params):
    rows, vocab, draws = 64, 32000, 4
    lg = _logits(rows, vocab, 7)
    hist = torch.randint(0, vocab, (rows, 40), generator=torch.Generator().manual_seed(9))
    dev = DeviceSampler(params, rows, vocab, range(100, 100 + rows), "cuda", history_len=64)
    dev.set_history(hist)
    host_rng = [SamplerRng(100 + b) for b in range(rows)]
    exact_rng = [SamplerRng(100 + b) for b in range(rows)]
    agree_host = agree_exact = total = 0
    lgc = lg.cuda()
    for _ in range(draws):
        got = dev.sample(lgc).cpu().tolist()
        for b in range(rows):
            agree_host += int(got[b] == sample_row(lg[b], params, hist[b].tolist(), host_rng[b]))
            agree_exact += int(got[b] == _exact_pick(lg[b], params, hist[b].tolist(), exact_rng[b].next_uniform()))
            total += 1
    # same RNG stream and ranking as the host policy. Against the policy evaluated in float64 only a
    # draw within ~1e-7 of one of the 32000 CDF boundaries can differ; the host's float32 running sum
    # is coarser than that in the low-probability tail, so agreement with it is lower there.
    assert agree_exact >= 0.97 * total, f"exact {agree_exact}/{total}"
    assert agree_host >= 0.7 * total, f"host {agree_host}/{total}"
    again = DeviceSampler(params, rows, vocab, range(100, 100 + rows), "cuda", history_len=64)
    again.set_history(hist)
    first = again.sample(lgc).cpu()
    ref = DeviceSampler(params, rows, vocab, range(100, 100 + rows), "cuda", history_len=64)
    ref.set_history(hist)
    assert torch.equal(first, ref.sample(lgc).cpu())


def _exact_pick(row, params, recent, u):
    """The sampling policy in float64 with the uniform draw ``u`` given."""
    x = row.clone()
    if params.repetition_penalty > 1.0:
        for t in recent[-params.repetition_window:]:
            x[t] = x[t] / params.repetition_penalty if x[t] > 0 else x[t] * params.repetition_penalty
    p = torch.softmax(x.double() / params.temperature, -1)
    order = torch.argsort(p, descending=True, stable=True)
    ps = p[order]
    cut = len(ps)
    if params.top_k > 0:
        cut = min(cut, params.top_k)
    if params.top_p < 1.0:
        cum = torch.cumsum(ps[:cut], 0)
        hit = torch.nonzero(cum >= params.top_p)
        if len(hit):
            cut = int(hit[0]) + 1
    cdf = torch.cumsum(ps[:cut], 0)
    r = int(torch.searchsorted(cdf, torch.tensor(u * float(cdf[-1]), dtype=torch.float64), right=True))
    return int(order[min(r, cut - 1)])


def test_empirical_distribution_follows_softmax():
    vocab, n = 8, 4096
    lg = torch.tensor([[2.0, 1.0, 0.5, 0.0, -0.5, -1.0, -2.0, -3.0]]).repeat(n, 1)
    s = DeviceSampler(SamplingParams(temperature=1.0), n, vocab, range(n), "cuda")
    tok = s.sample(lg.cuda()).cpu()
    freq = torch.bincount(tok, minlength=vocab).float() / n
    p = torch.softmax(lg[0], -1)
    assert (freq - p).abs().max().item() < 0.03


def test_engine_sampled_generation_graph_equals_eager():
    cfg = SciAgentConfig(vocab_size=512, d_model=256, n_layers=2, n_heads=4, n_kv_heads=2, d_ff=512, max_seq_len=256)
    model = GQADecoder(cfg, device="cuda", seed=5, init_std=0.08)
    prompts = torch.randint(0, 512, (3, 20), generator=torch.Generator().manual_seed(2))
    params = SamplingParams(temperature=0.9, top_k=40, top_p=0.95, repetition_penalty=1.1)
    a = InferenceEngine(model, max_batch=3, max_seq=64, page=16, use_graph=True).generate(prompts, 12, params, seed=11)
    b = InferenceEngine(model, max_batch=3, max_seq=64, page=16, use_graph=False).generate(prompts, 12, params, seed=11)
    assert torch.equal(a.cpu(), b.cpu())
    c = InferenceEngine(model, max_batch=3, max_seq=64, page=16).generate(prompts, 12, params, seed=12)
    assert not torch.equal(a.cpu(), c.cpu())


@pytest.mark.parametrize("vocab", [5, 8192, 8193, 100003, 128256, 393221])
def test_equal_logits_take_ties_in_id_order_on_every_row_split(vocab):
    """All weights equal: the draw is the floor(u * V)-th id, wherever the row is cut (one CTA, eight CTAs with a slice
    in shared memory, a slice too long for it); a row with one id masked shifts every id behind it by one."""
    rows = 5
    lg = torch.zeros(rows, vocab)
    hole = vocab // 3
    lg[rows - 1, hole] = float("-inf")
    s = DeviceSampler(SamplingParams(temperature=1.0), rows, vocab, range(50, 50 + rows), "cuda")
    got = s.sample(lg.cuda()).cpu().tolist()
    w = 2 ** 32 - 1
    for b in range(rows):
        n = vocab - (b == rows - 1)
        z = n * w
        t = min(int(SamplerRng(50 + b).next_uniform() * float(z)), z - 1)
        want = t // w
        if b == rows - 1 and want >= hole:
            want += 1
        assert got[b] == want


@pytest.mark.parametrize("vocab", [1, 37, 8191, 20001])
def test_odd_rows_and_penalties_match_the_float64_policy(vocab):
    """Odd lengths (unaligned rows), a window with repeats, top-k and top-p together: only a draw within rounding of a
    CDF boundary may differ from the float64 statement."""
    rows = 32
    params = SamplingParams(temperature=0.8, top_k=40, top_p=0.9, repetition_penalty=1.3, repetition_window=8)
    lg = _logits(rows, vocab, 21)
    hist = torch.randint(0, vocab, (rows, 12), generator=torch.Generator().manual_seed(3))
    hist[:, 9] = hist[:, 7]
    dev = DeviceSampler(params, rows, vocab, range(rows), "cuda", history_len=16)
    dev.set_history(hist)
    got = dev.sample(lg.cuda()).cpu().tolist()
    same = sum(got[b] == _exact_pick(lg[b], params, hist[b].tolist(), SamplerRng(b).next_uniform()) for b in range(rows))
    assert same >= rows - 1


def _greedy_pick(row, recent, penalty):
    """First maximum of the penalised row; a NaN never beats a number, but one in column 0 is never displaced."""
    v, p = row.clone(), torch.tensor(penalty, dtype=torch.float32)
    for t in recent:
        if 0 <= t < len(v):
            v[t] = v[t] / p if v[t] > 0 else v[t] * p
    if v[0] != v[0]:
        return 0
    v = v.masked_fill(v != v, float("-inf"))
    return int((v == v.max()).nonzero()[0])


@pytest.mark.parametrize("vocab", [1, 3, 2047, 2049, 4097, 8191, 16384, 16389, 100003, 600001])
@pytest.mark.parametrize("rows", [1, 20, 64])
@pytest.mark.parametrize("penalty", [1.0, 1.5])
def test_greedy_rows_on_every_split(vocab, rows, penalty):
    """One CTA per row and clusters of two to eight, rows at any alignment: ties at the first and last element of a slice, NaN in
    column 0 and elsewhere, rows of -inf only, and windows that repeat the winner or share its bit of the bitmap."""
    wide = torch.randn(rows, vocab + 3, generator=torch.Generator().manual_seed(vocab)).cuda()
    lg = wide[:, :vocab]
    hist = torch.randint(0, vocab, (rows, 16), generator=torch.Generator().manual_seed(2))
    for b in range(rows):
        top = int(lg[b].argmax())
        hist[b, 3] = hist[b, 9] = top
        hist[b, 5] = (top + 65536) % vocab
        cut = ((vocab + 3) // 4 + 3) // 4 * 4
        if b % 5 == 1:
            lg[b, vocab - 1] = lg[b, min(cut, vocab - 1)] = lg[b, max(min(cut, vocab) - 1, 0)] = 9.0
        if b % 5 == 2:
            lg[b, vocab // 2:] = float("nan")
        if b % 5 == 3:
            lg[b] = float("-inf")
        if b % 5 == 4:
            lg[b, 0] = float("nan")
    s = DeviceSampler(SamplingParams(temperature=0.0, repetition_penalty=penalty, repetition_window=12), rows, vocab,
                      range(rows), "cuda", history_len=16)
    s.set_history(hist)
    got = s.sample(lg).cpu().tolist()
    host = lg.cpu()
    want = [_greedy_pick(host[b], hist[b, 4:].tolist() if penalty > 1 else [], penalty) for b in range(rows)]
    assert got == want


@pytest.mark.parametrize("vocab", [700, 8200, 128256, 393221])
@pytest.mark.parametrize("ties", [1, 511, 512, 513, 640])
@pytest.mark.parametrize("top_k,top_p", [(0, 1.0), (0, 0.5), (1, 1.0), (512, 1.0), (600, 0.7)])
def test_short_lists_and_walks_take_the_same_element(vocab, ties, top_k, top_p):
    """`ties` ids share the largest weight and the rest are masked: up to 512 of them are finished as a list by one CTA, more
    by the walks. The kept set is a prefix of the ids and the draw an exact integer statement either way."""
    rows = 3
    ids = torch.stack([torch.randperm(vocab, generator=torch.Generator().manual_seed(ties + b))[:ties].sort().values
                       for b in range(rows)])
    lg = torch.full((rows, vocab), float("-inf")).scatter_(1, ids, 0.0)
    params = SamplingParams(temperature=1.0, top_k=top_k, top_p=top_p)
    s = DeviceSampler(params, rows, vocab, range(7, 7 + rows), "cuda")
    got = s.sample(lg.cuda()).cpu().tolist()
    w = 2 ** 32 - 1
    for b in range(rows):
        kept = min(ties, top_k) if 0 < top_k < vocab else ties
        if top_p < 1.0:                           # the first prefix whose weight reaches top_p of the total
            kept = min(kept, -(-math.ceil(float(torch.tensor(top_p)) * float(ties * w)) // w))
        z = kept * w
        t = min(int(SamplerRng(7 + b).next_uniform() * float(z)), z - 1)
        assert got[b] == int(ids[b, t // w])


@pytest.mark.parametrize("vocab", [8193, 32000, 100003, 128256])
@pytest.mark.parametrize("rows", [16, 34, 64, 150])
@pytest.mark.parametrize("params", [SamplingParams(temperature=0.8, top_k=50, top_p=0.95), SamplingParams(temperature=1.1),
                                    SamplingParams(temperature=0.7, top_k=700, top_p=0.9, repetition_penalty=1.3)])
def test_batches_draw_what_their_rows_draw_alone(vocab, rows, params):
    """A row's CTAs are fewer in a batch whose clusters of eight do not all run at once. Sums are of integers, so a row of the batch
    draws the same token, and leaves the same generator, as alone on a cluster of eight."""
    lg = _logits(rows, vocab, vocab + rows).cuda()
    hist = torch.randint(0, vocab, (rows, 40), generator=torch.Generator().manual_seed(rows))
    seeds = list(range(50, 50 + rows))
    batch = DeviceSampler(params, rows, vocab, seeds, "cuda", history_len=64)
    batch.set_history(hist)
    got = batch.sample(lg).tolist()
    for b in range(0, rows, 7):
        one = DeviceSampler(params, 1, vocab, seeds[b:b + 1], "cuda", history_len=64)
        one.set_history(hist[b:b + 1])
        assert one.sample(lg[b:b + 1]).tolist() == got[b:b + 1]
        assert torch.equal(one.state, batch.state[b:b + 1])
