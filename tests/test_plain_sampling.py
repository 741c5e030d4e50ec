"""The plain selection itself (no GPU)."""
import pytest
import torch

import plain_sampling as ps


def test_philox_known_answer():
    # Philox4x32-10 with an all-zero counter and key (first word of the published test vector)
    assert ps.philox_first_word(0, 0) == 0x6627E8D5
    assert 0.0 < ps.uniform(3, 5) < 1.0 and ps.uniform(3, 5) != ps.uniform(3, 6) != ps.uniform(4, 5)


def test_filters():
    l = torch.tensor([0.0, 3.0, 1.0, 2.0, -1.0])
    assert ps.sample(l, 0.0)[0] == 1
    assert all(ps.sample(l, 1.0, top_k=1, seed=s)[0] == 1 for s in range(20))
    assert {ps.sample(l, 1.0, top_k=2, seed=s)[0] for s in range(200)} == {1, 3}
    # softmax(l) = [.03, .64, .09, .24, .01]: p = 0.7 keeps {1, 3}; p = 0.5 keeps {1}
    assert {ps.sample(l, 1.0, top_p=0.7, seed=s)[0] for s in range(200)} == {1, 3}
    assert {ps.sample(l, 1.0, top_p=0.5, seed=s)[0] for s in range(50)} == {1}
    # penalty 4 on token 1: 3.0 -> 0.75; on token 4: -1 -> -4
    out = ps.penalise(l, [1, 4, 1], 4.0)
    assert out.tolist() == [0.0, 0.75, 1.0, 2.0, -4.0]
    assert ps.sample(l, 0.0, repetition_penalty=4.0, generated=[1])[0] == 3
    tok, acceptable, cut = ps.sample(l, 1.0, top_p=0.7, seed=1)
    assert acceptable == {tok} and cut > 0.01


def test_sampler_packs_the_rows_parameters_into_one_buffer():
    """The sampler's per-row parameters travel as one buffer of 4-byte words (seeds and token
    counters as 64-bit values first, so that they stay aligned); the views handed to the kernel
    must read back what went in, also when the ring of host buffers comes round."""
    from nanoinfer_b200.sampling import Sampler, SamplingParams
    s = Sampler(vocab_size=100, device=torch.device("cpu"))
    for n in (1, 3, 5, 70):                          # 70 rows outgrow the first buffer
        params = [SamplingParams(temperature=0.5 + r, top_k=r - 1, top_p=1.0 / (r + 1)) for r in range(n)]
        seeds = [(1 << 55) - 1 - r for r in range(n)]
        counts = list(range(10, 10 + n))
        for _ in range(6):                           # more calls than host buffers
            seed_t, count_t, temp_t, top_p_t, top_k_t = s._upload(torch.device("cpu"), params, seeds, counts)
            assert seed_t.dtype == torch.int64 and seed_t.tolist() == seeds
            assert count_t.dtype == torch.int64 and count_t.tolist() == counts
            assert temp_t.dtype == torch.float32 and temp_t.tolist() == [0.5 + r for r in range(n)]
            assert torch.allclose(top_p_t, torch.tensor([1.0 / (r + 1) for r in range(n)]))
            assert top_k_t.dtype == torch.int32 and top_k_t.tolist() == [r - 1 for r in range(n)]
    assert s.h2d_bytes == 6 * 28 * (1 + 3 + 5 + 70)


@pytest.mark.parametrize("rows", [3, 70])
def test_parameters_are_packed_once_whichever_way_they_travel(rows, monkeypatch):
    """A vocabulary or a batch that does not take them with the launch gets the same words by the copy."""
    from nanoinfer_b200.kernels import ops
    from nanoinfer_b200.sampling import Sampler, SamplingParams
    params = [SamplingParams(temperature=0.5 + r, top_k=r, top_p=0.25, seed=r) for r in range(rows)]
    seeds, at = [2 ** 63 + r for r in range(rows)], [5 - r for r in range(rows)]
    for offered in (False, True):
        sampler, packs, drawn, taken = Sampler(100, torch.device("cpu")), [], [], []
        words = sampler._words
        monkeypatch.setattr(sampler, "_words", lambda *a: packs.append(words(*a)) or packs[-1])
        monkeypatch.setattr(ops, "sample_values", lambda logits, out, w: taken.append(w) is None and offered)
        monkeypatch.setattr(ops, "sample", lambda logits, out, t, k, p, s, c: drawn.append((t.tolist(), k.tolist(), p.tolist(), s.tolist(), c.tolist())))
        monkeypatch.setattr(ops, "current_stream_object", lambda: None)
        sampler.sample(torch.zeros(rows, 100), params, seeds, at)
        assert len(packs) == 1 and len(packs[0]) == 28 * rows == sampler.h2d_bytes and taken == packs
        want = ([p.temperature for p in params], [p.top_k for p in params], [0.25] * rows, [s - 2 ** 64 for s in seeds], at)
        assert drawn == ([] if offered else [want])
