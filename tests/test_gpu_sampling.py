"""The sampling kernels against the plain selection, row by row."""
import pytest
import torch

import plain_sampling as ps

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _logits(rows, vocab, seed, scale=3.0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(rows, vocab, generator=g) * scale


@pytest.mark.parametrize("vocab", [256, 1000, 128256])
def test_argmax_ties_go_to_the_lowest_id(vocab):
    from nanoinfer_b200.kernels import ops
    l = _logits(5, vocab, 0)
    l[1, 7] = l[1, vocab - 3] = l[1].max() + 1.0     # a tie: the lower id wins
    l[2, :] = 0.5                                    # all equal: id 0
    l[3, vocab - 1] = 100.0                          # the last id
    out = torch.empty(5, dtype=torch.int32, device=DEV)
    ops.argmax(l.to(DEV), out)
    want = [int(torch.argmax(l[0])), 7, 0, vocab - 1, int(torch.argmax(l[4]))]
    assert out.tolist() == want


CASES = [dict(temperature=1.0), dict(temperature=0.7), dict(temperature=1.5, top_k=5),
         dict(temperature=0.8, top_p=0.9), dict(temperature=1.0, top_k=40, top_p=0.5),
         dict(temperature=0.0), dict(temperature=1.0, top_k=1), dict(temperature=2.0, top_p=0.05),
         dict(temperature=0.9, repetition_penalty=1.3), dict(temperature=0.0, repetition_penalty=2.0)]


@pytest.mark.parametrize("vocab", [4096, 5001, 33007, 128256, 262145])
def test_a_cluster_per_row_selects_the_same_tokens_as_one_block(vocab):
    """Rows of every kind of parameters, at vocabularies that do and do not divide by the cluster's
    eight blocks: the cluster kernel and the one-block kernel agree on every token, bit for bit."""
    from nanoinfer_b200.kernels import ops
    rows = 40
    g = torch.Generator().manual_seed(vocab)
    l = (torch.randn(rows, vocab, generator=g) * 3.0).to(DEV)
    l[3] = 0.25                                                     # all equal: every id as likely
    l[4, :] = -0.0
    l[4, 17] = 0.0                                                  # +0 and -0 tie: the lowest id wins a greedy row
    temps = torch.tensor([[0.0, 0.7, 1.0, 1.5][i % 4] for i in range(rows)], device=DEV)
    temps[4] = 0.0
    ks = torch.tensor([[0, 1, 40, 5000, vocab, 0][i % 6] for i in range(rows)], dtype=torch.int32, device=DEV)
    ps_ = torch.tensor([[1.0, 0.9, 0.5, 0.05, 0.999][i % 5] for i in range(rows)], device=DEV)
    seeds = torch.arange(rows, dtype=torch.int64, device=DEV) * 7919
    counters = torch.arange(rows, dtype=torch.int64, device=DEV) % 5
    outs = []
    for cluster in (True, False):
        ops.sample_by_cluster(cluster)
        out = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
        ops.sample(l, out, temps, ks, ps_, seeds, counters)
        outs.append(out.cpu())
    ops.sample_by_cluster(True)
    assert torch.equal(outs[0], outs[1]), f"rows {torch.nonzero(outs[0] != outs[1]).flatten().tolist()} differ"
    assert int(outs[0].min()) >= 0 and int(outs[0].max()) < vocab and int(outs[0][4]) == 0
    # many draws of one row: different counters give different tokens, the same counter the same token
    many = 64
    rep = l[1:2].expand(many, vocab).contiguous()
    out_a = torch.empty(many, dtype=torch.int32, device=DEV)
    t1 = torch.ones(many, device=DEV)
    z0 = torch.zeros(many, dtype=torch.int32, device=DEV)
    sd = torch.full((many,), 5, dtype=torch.int64, device=DEV)
    ops.sample(rep, out_a, t1, z0, t1, sd, torch.arange(many, dtype=torch.int64, device=DEV))
    assert len(set(out_a.tolist())) > many // 2
    out_b = torch.empty_like(out_a)
    ops.sample(rep, out_b, t1, z0, t1, sd, torch.zeros(many, dtype=torch.int64, device=DEV))
    assert len(set(out_b.tolist())) == 1 and out_b[0] == out_a[0]


def _tied_rows(vocab, ties, rows, seed):
    """40 tokens at 5, ``ties`` per eighth of the row at 4, the rest far below."""
    g = torch.Generator().manual_seed(seed)
    l = torch.randn(rows, vocab, generator=g) - 50.0
    for r in range(rows):
        for c in range(8):
            lo, hi = c * vocab // 8, (c + 1) * vocab // 8
            l[r, lo + torch.randperm(hi - lo, generator=g)[:ties]] = 4.0
        l[r, torch.randperm(vocab, generator=g)[:40]] = 5.0
    return l


@pytest.mark.parametrize("vocab, ties", [(4104, 20), (4104, 33), (33000, 120), (33000, 480), (128256, 250), (128256, 495)])
def test_top_k_with_thousands_tied_at_the_kth_place(vocab, ties):
    """All tokens that tie with the k-th stay: from a few more than are compared pair by pair to thousands; probabilities that
    tie at the top-p place too, one that takes a few of them, temperatures that round most masses to zero."""
    from nanoinfer_b200.kernels import ops
    rows = 12
    l = _tied_rows(vocab, ties, rows, vocab + ties)
    l[1] += torch.rand(vocab, generator=torch.Generator().manual_seed(1)) * 1e-6 * (l[1] > 4.5)           # masses that differ in the last bits
    l[2, l[2] == 4.0] = -40.0                                                                              # tied at a mass of nearly nothing
    l = l.to(DEV)
    k_t = torch.tensor([41 + 3 * (r % 3) for r in range(rows)], dtype=torch.int32, device=DEV)
    seeds, counters = torch.arange(rows, device=DEV) * 104729, torch.arange(rows, device=DEV) % 3
    for temp, p in [(0.8, 1.0), (0.8, 0.9), (0.8, 0.05), (0.03, 0.9999), (0.004, 0.9), (3.0, 0.5)]:
        temps, ps_ = torch.full((rows,), temp, device=DEV), torch.full((rows,), p, device=DEV)
        outs = []
        for cluster in (True, False):
            ops.sample_by_cluster(cluster)
            out = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
            ops.sample(l, out, temps, k_t, ps_, seeds, counters)
            outs.append(out.cpu())
        ops.sample_by_cluster(True)
        assert torch.equal(outs[0], outs[1]), (temp, p)


def test_tied_rows_take_no_comparisons_of_all_pairs():
    """Thousands of tied tokens may cost passes over them (as long as a row without candidates, about five times the plain
    row's), not a comparison of each with each (about sixty times)."""
    from nanoinfer_b200.kernels import ops
    rows, vocab = 8, 128256

    def best_of(l):
        l = l.to(DEV)
        out = torch.empty(rows, dtype=torch.int32, device=DEV)
        k_t, ps_ = torch.full((rows,), 50, dtype=torch.int32, device=DEV), torch.full((rows,), 0.9, device=DEV)
        temps, seeds = torch.full((rows,), 0.8, device=DEV), torch.arange(rows, device=DEV)
        times = []
        for _ in range(20):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                ops.sample(l, out, temps, k_t, ps_, seeds, seeds)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    plain, tied = best_of(torch.randn(rows, vocab, generator=torch.Generator().manual_seed(2)) * 3), best_of(_tied_rows(vocab, 490, rows, 3))
    assert tied < 15 * plain, (tied, plain)


@pytest.mark.parametrize("vocab", [4096, 4097, 33000, 128256])
def test_top_k_from_candidates_selects_the_same_tokens_as_one_block(vocab):
    """Rows with top-k whose blocks send a few candidates, and rows that send too many (large k, equal logits, most of a row
    masked with -inf) and go the general way: k from 1 to beyond what a block may send, ties at the k-th place and among the
    probabilities, logits that differ only far behind the leading bits, negative rows, masked rows, with and without top-p."""
    from nanoinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(vocab)
    ks = [1, 2, 50, 200, 503, 505, 3000, vocab - 1]
    tops = [1.0, 0.9, 0.3, 0.9999999]
    kinds = 8
    rows = kinds * len(ks)
    l = torch.randn(rows, vocab, generator=g) * 3.0
    for i in range(len(ks)):
        l[kinds * i + 1] = (l[kinds * i + 1] * 2).round() / 2                       # many ties
        l[kinds * i + 2] = 0.25                                                     # all equal
        l[kinds * i + 3] = 5.0 + torch.rand(vocab, generator=g) * 1e-4              # one leading value, different tails
        l[kinds * i + 4] = -100.0 + l[kinds * i + 4]                                # all negative
        l[kinds * i + 5, torch.randperm(vocab, generator=g)[: vocab - 120]] = -float("inf")      # masked but for 120 tokens
        l[kinds * i + 6] = l[kinds * i + 6].abs().neg().mul(50)                     # probabilities that round to a mass of zero
        l[kinds * i + 7, :vocab // 8] += 30.0                                       # everything that counts in the first block's slice
    l = l.to(DEV)
    k_t = torch.tensor([ks[r // kinds] for r in range(rows)], dtype=torch.int32, device=DEV)
    seeds = torch.arange(rows, dtype=torch.int64, device=DEV) * 7919
    counters = torch.arange(rows, dtype=torch.int64, device=DEV) % 5
    temps = torch.tensor([[0.7, 1.0, 1.5][r % 3] for r in range(rows)], device=DEV)
    for p in tops:
        ps_ = torch.full((rows,), p, device=DEV)
        outs = []
        for cluster in (True, False):
            ops.sample_by_cluster(cluster)
            out = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
            ops.sample(l, out, temps, k_t, ps_, seeds, counters)
            outs.append(out.cpu())
        ops.sample_by_cluster(True)
        assert torch.equal(outs[0], outs[1]), f"rows {torch.nonzero(outs[0] != outs[1]).flatten().tolist()} differ at top-p {p}"


@pytest.mark.parametrize("vocab", [384, 1000, 128256])
def test_sampler_matches_plain_selection(vocab):
    from nanoinfer_b200.sampling import Sampler, SamplingParams
    sampler = Sampler(vocab, torch.device(DEV))
    rows = len(CASES) * 3
    l = _logits(rows, vocab, 1)
    params, seeds, idxs, gens = [], [], [], []
    for r in range(rows):
        c = CASES[r % len(CASES)]
        params.append(SamplingParams(**c))
        seeds.append(1000 + r // len(CASES))
        idxs.append(r)
        g = torch.Generator().manual_seed(r)
        gens.append(torch.randint(0, vocab, (20,), generator=g).tolist() + [int(torch.argmax(l[r]))])
    got = sampler.sample(l.clone().to(DEV), params, seeds, idxs, gens).tolist()
    skipped = 0
    for r in range(rows):
        p = params[r]
        tok, acceptable, cut_margin = ps.sample(l[r], p.temperature, p.top_k, p.top_p, p.repetition_penalty,
                                                gens[r], seeds[r], idxs[r])
        if cut_margin < ps.ROUNDING:      # the top-p cut itself is within rounding: two valid kept sets
            skipped += 1
            continue
        assert got[r] in acceptable, f"row {r} {p}: kernel {got[r]}, plain {tok} (acceptable {acceptable})"
    assert skipped <= 1


def test_draws_follow_the_distribution_and_do_not_depend_on_the_batch():
    from nanoinfer_b200.sampling import Sampler, SamplingParams
    vocab, n = 12, 6000
    sampler = Sampler(vocab, torch.device(DEV))
    row = torch.tensor([2.0, 1.0, 0.0, -1.0, 0.5, 1.5, -3.0, 0.0, 0.2, 1.1, -0.5, 0.7])
    l = row.repeat(n, 1)
    sp = SamplingParams(temperature=0.8, seed=5)
    got = sampler.sample(l.to(DEV), [sp] * n, [5] * n, list(range(n))).cpu()
    probs = torch.softmax(row / 0.8, 0)
    freq = torch.bincount(got.long(), minlength=vocab).double() / n
    sigma = torch.sqrt(probs * (1 - probs) / n)
    assert torch.all((freq - probs).abs() <= 5 * sigma + 1e-9)
    # token i of a request is the same alone, in another row, or beside other requests
    alone = sampler.sample(row[None].to(DEV), [sp], [5], [17]).item()
    assert alone == got[17].item()
    mixed = sampler.sample(l[:3].to(DEV), [SamplingParams.greedy(), sp, SamplingParams(seed=9)], [0, 5, 9], [0, 17, 3])
    assert mixed[1].item() == alone and mixed[0].item() == 0


@pytest.mark.parametrize("vocab", [4096, 4100, 6000, 16384, 16388, 50257, 128256])
def test_candidates_of_rows_of_every_range(vocab):
    """What the slices send as candidates of a row with top-k depends on the range of its logits: signed zeros, rows around
    zero, rows of huge and of tiny spread, one far token, infinities, short last slices, slices of fewer than k tokens."""
    from nanoinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(vocab)
    base = torch.randn(vocab, generator=g)
    far, most, zeros = base.clone(), torch.full((vocab,), torch.finfo(torch.float32).min), torch.zeros(vocab)
    far[vocab // 3] = 1e30
    most[torch.randperm(vocab, generator=g)[:700]] = base[:700]
    zeros[torch.randperm(vocab, generator=g)[:vocab // 2]] *= -1.0
    zeros[torch.randperm(vocab, generator=g)[:30]] = base[:30]
    last = base.clone()
    last[-100:] += 40.0
    inf = base.clone()
    inf[5] = float("inf")
    rows = [base, base * 1e-30, base * 1e30, base - 3.0, base * 0.1 - 1.0, far, most, zeros, last, -base.abs(), inf, base.round()]
    l = torch.stack(rows).to(DEV)
    n = len(rows)
    seeds, counters = torch.arange(n, device=DEV) * 31 + 7, torch.arange(n, device=DEV)
    temps = torch.full((n,), 0.9, device=DEV)
    for k in (1, 50, 300, 504, 505):
        for p in (1.0, 0.9):
            outs = []
            for cluster in (True, False):
                ops.sample_by_cluster(cluster)
                out = torch.full((n,), -1, dtype=torch.int32, device=DEV)
                ops.sample(l, out, temps, torch.full((n,), k, dtype=torch.int32, device=DEV), torch.full((n,), p, device=DEV), seeds, counters)
                outs.append(out.tolist())
            ops.sample_by_cluster(True)
            assert outs[0] == outs[1], (k, p)


@pytest.mark.parametrize("rows, vocab, taken", [(1, 4096, True), (64, 4096, True), (65, 4096, False), (3, 4095, False), (2, 400000, False)])
def test_parameters_that_travel_with_the_launch(rows, vocab, taken):
    """The same tokens whether a batch's parameters are arguments of the launch or arrays on the device."""
    import struct
    from nanoinfer_b200.kernels import ops
    from nanoinfer_b200.sampling import Sampler, SamplingParams
    g = torch.Generator().manual_seed(rows)
    l = (torch.randn(rows, vocab, generator=g) * 3).to(DEV)
    params = [SamplingParams(temperature=[0.7, 0.0, 1.3][r % 3], top_k=[-1, 20, 300][r % 3 if r % 2 else 0], top_p=[0.9, 1.0][r % 2]) for r in range(rows)]
    seeds, at = [2 ** 63 + r for r in range(rows)], [5 * r for r in range(rows)]
    words = struct.pack(f"<{rows}Q{rows}q{rows}f{rows}f{rows}i", *seeds, *at, *(p.temperature for p in params), *(p.top_p for p in params),
                        *(p.top_k for p in params))
    out, want = torch.full((rows,), -1, dtype=torch.int32, device=DEV), torch.full((rows,), -1, dtype=torch.int32, device=DEV)
    assert ops.sample_values(l, out, words) == taken
    sampler = Sampler(vocab, torch.device(DEV))
    s, c, t, p, k = sampler._upload(l.device, params, seeds, at)
    ops.sample(l, want, t, k, p, s, c)
    assert not taken or torch.equal(out, want)
    assert torch.equal(sampler.sample(l, params, seeds, at), want)
    assert sampler.h2d_bytes == 2 * 28 * rows


def _sample_us(logits, k, top_p=0.9):
    """Microseconds of one call, by itself in a graph of twenty."""
    from nanoinfer_b200.kernels import ops
    n = logits.shape[0]
    out = torch.empty(n, dtype=torch.int32, device=DEV)
    rows = torch.arange(n, dtype=torch.int64, device=DEV)
    args = (torch.full((n,), 0.8, device=DEV), torch.full((n,), k, dtype=torch.int32, device=DEV), torch.full((n,), top_p, device=DEV), rows, rows)
    ops.sample(logits, out, *args)
    graph, start, end = torch.cuda.CUDAGraph(), torch.cuda.Event(True), torch.cuda.Event(True)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        for _ in range(20):
            ops.sample(logits, out, *args)
    times = []
    for _ in range(4):
        start.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end) * 50)
    return min(times)


@pytest.mark.parametrize("spread", ["normal", "uniform"])
def test_a_large_k_stays_with_the_candidates(spread):
    """Up to a k near what a slice can send, a row goes by its candidates: 8 rows of 128,256 take 35 to 43 us for k = 320 to 490, where
    passes over the row take 103 to 130."""
    g = torch.Generator().manual_seed(3)
    l = (torch.randn(8, 128256, generator=g) * 3 if spread == "normal" else torch.rand(8, 128256, generator=g) * 10).to(DEV)
    passes = _sample_us(l, 600)                      # more than a slice can send
    for k in (289, 320, 350, 400, 490):
        assert _sample_us(l, k) < 0.6 * passes, k


@pytest.mark.parametrize("k", [288, 289, 320, 400, 490, 504, 505])
@pytest.mark.parametrize("vocab", [16384, 50257, 128256])
def test_a_large_k_draws_the_same_tokens(vocab, k):
    from nanoinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(k)
    l = torch.randn(8, vocab, generator=g) * 3
    l[1] = (l[1] * 2).round() / 2                    # ties
    l[2] = torch.rand(vocab, generator=g)
    l[3, torch.randperm(vocab, generator=g)[: vocab - 450]] = -float("inf")          # fewer tokens than k, or little more
    l[4, : vocab // 8] += 30.0                       # all in the first block's slice
    l[5, 7] = 1e30
    l[6] = l[6].abs().neg()
    l = l.to(DEV)
    rows = torch.arange(8, dtype=torch.int64, device=DEV)
    for p in (0.9, 1.0):
        outs = []
        for cluster in (True, False):
            ops.sample_by_cluster(cluster)
            out = torch.full((8,), -1, dtype=torch.int32, device=DEV)
            ops.sample(l, out, torch.full((8,), 0.9, device=DEV), torch.full((8,), k, dtype=torch.int32, device=DEV), torch.full((8,), p, device=DEV), rows, rows)
            outs.append(out.tolist())
        ops.sample_by_cluster(True)
        assert outs[0] == outs[1], p


@pytest.mark.parametrize("tied", [40, 256, 257, 300, 511, 512, 513, 700, 2000, 3900])
@pytest.mark.parametrize("others", [0, 3])
def test_tokens_of_one_value_at_the_k_th_place(tied, others):
    """All of the k-th's coarse value are one number (they stay unlooked at), or a few beside them differ in their last bits."""
    from nanoinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(tied)
    l = torch.randn(4, 128256, generator=g)
    for r in range(4):
        at = torch.randperm(128256, generator=g)
        l[r, at[:30]] = 9.0 + torch.rand(30, generator=g)
        l[r, at[30:30 + tied]] = 8.0
        for i in range(others):
            l[r, at[100 + tied + i]] = torch.nextafter(torch.tensor(8.0), torch.tensor(9.0 if i % 2 else 7.0)).item()
    l = l.to(DEV)
    rows = torch.arange(4, dtype=torch.int64, device=DEV)
    for p in (0.95, 1.0):
        outs = []
        for cluster in (True, False):
            ops.sample_by_cluster(cluster)
            out = torch.full((4,), -1, dtype=torch.int32, device=DEV)
            ops.sample(l, out, torch.full((4,), 1.5, device=DEV), torch.full((4,), 50, dtype=torch.int32, device=DEV), torch.full((4,), p, device=DEV), rows, rows)
            outs.append(out.tolist())
        ops.sample_by_cluster(True)
        assert outs[0] == outs[1], p
