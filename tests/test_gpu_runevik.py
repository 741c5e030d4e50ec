"""Runevik on the GPU against the plain implementation (tests/plain_runevik.py): every mechanism alone, then
whole models replayed under four ways of cutting the same requests - in 32-bit and in bfloat16 - and greedy
generation through the engine.  The models are small, of other sizes than any real one, with weights tuned
so that a lost key, a lost state or a shifted convolution tap moves the logits far beyond rounding."""
import copy

import pytest
import torch

import replay_util as ru
import tiny_runevik as tr
from helpers import load_plain, random_tokens
from plain_runevik import (PlainRunevik, delta_mixer, delta_state, gelu_tanh, over_rms, sinusoid)

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
CUTS = {"whole": ru.whole, "tail": ru.tail_by_token, "ragged": ru.ragged, "mixed": ru.mixed}
LENGTHS = {"r1": [1, 2, 17, 33, 70, 130, 49], "r2": [3, 16, 64, 150, 31, 97], "r3": [2, 48, 129, 15, 80]}
RAW = {"r1": tr.R1, "r2": tr.R2, "r3": tr.R3}


def _keep_state(tensors):
    """Decays close to one, so that what a delta layer wrote hundreds of tokens ago still counts."""
    for name, t in tensors.items():
        if name.endswith("mix.A_log"):
            t.fill_(-4.0)
        if name.endswith(".norm1") or name == "final.norm":
            t.fill_(1.25)
        if name.endswith("mix.norm") or name.endswith("side.norm") or name.endswith("dkv.norm"):
            t.copy_((1.0 + 0.3 * torch.randn(t.shape, generator=torch.Generator().manual_seed(t.numel()))).to(t.dtype))


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    """{key: (folder, config dictionary, requests, plain logits per request)}"""
    root = tmp_path_factory.mktemp("runevik")
    out = {}
    for seed, (key, raw) in enumerate(RAW.items()):
        d = str(root / key)
        tr.write_model(d, raw, seed + 11, tune=_keep_state)
        cfg, w = load_plain(d)
        plain = PlainRunevik(cfg, w)
        reqs = {f"q{i}": random_tokens(raw["vocab"], n, 31 * seed + i) for i, n in enumerate(LENGTHS[key])}
        want = {rid: plain.run(toks, plain.new_state())[0].float() for rid, toks in reqs.items()}
        out[key] = (d, cfg, reqs, want)
        SENSITIVITY[key] = _sensitivity(cfg, w, reqs, want)
    return out


SENSITIVITY = {}


def _sensitivity(cfg, w, reqs, want):
    """How much more than the median position each position's logits move when every weight is disturbed at the
    size of a bfloat16 rounding: {(request, position): factor >= 1}.  Where the delta rule subtracts a good
    prediction, or a norm divides by a small mean, a position can be ten times as sensitive as most."""
    g = torch.Generator().manual_seed(0)
    moved = {}
    for trial in range(3):                       # a position's sensitivity depends on the direction: the largest of three
        shaken = {k: v.double() * (1 + 2.0 ** -8 * (torch.rand(v.shape, generator=g, dtype=torch.float64) - 0.5))
                  for k, v in w.items()}
        plain = PlainRunevik(cfg, shaken)
        for rid, toks in reqs.items():
            out = plain.run(toks, plain.new_state())[0].float()
            rel = (out - want[rid]).pow(2).mean(1).sqrt() / want[rid].pow(2).mean(1).sqrt()
            for pos in range(len(toks)):
                moved[(rid, pos)] = max(moved.get((rid, pos), 0.0), rel[pos].item())
    median = sorted(moved.values())[len(moved) // 2]
    return {k: max(1.0, v / (3.0 * median)) for k, v in moved.items()}


# bfloat16 bounds of the whole-model replays: per position twice those of the Llama replays (ru.compare), since a
# layer of this design rounds more often on the way to the stream - three normed sums (mixer output, feed-forward
# activation, token input) whose direction carries every rounding of their inputs at full weight.  And the delta
# rule subtracts what the state already predicts (the value minus what the state returns for its key): where the prediction is good, the difference is
# small and the roundings of its two terms are not, so single positions stand out.  Hence the rule: at most
# 3 % of the positions over the bound, none over four times the bound, and the bound of a position that is more
# than three times as sensitive as the median position (measured on the plain model, see _sensitivity) grows in
# proportion.  A lost key, state or tap moves these models' logits by more than that at most positions (the
# far-token tests, which keep the tight bounds, show it).
BF16_MAX_REL, BF16_RMS_REL, BF16_SHARE_OVER, BF16_WORST = 0.10, 0.03, 0.03, 4.0


def _compare(got, want, dtype, label, sensitivity=None):
    if dtype == "float32":
        return ru.compare(got, want, dtype, label)
    assert got
    ratios = {}
    for (rid, pos), row in got.items():
        ref = want[rid][pos]
        err = (row - ref).abs()
        ratios[(rid, pos)] = max(err.max().item() / (BF16_MAX_REL * ref.abs().max().item()),
                                 err.pow(2).mean().sqrt().item() / (BF16_RMS_REL * ref.pow(2).mean().sqrt().item())) \
            / (sensitivity or {}).get((rid, pos), 1.0)
    over = {k: round(v, 2) for k, v in ratios.items() if v > 1.0}
    worst = max(ratios.values())
    assert worst <= BF16_WORST, f"{label}: worst position at {worst:.2f} times the bound: {over}"
    assert len(over) <= max(1, BF16_SHARE_OVER * len(ratios)), f"{label}: {len(over)} of {len(ratios)} positions over the bound: {over}"


def _runner(model_dir, dtype, steps, page=16, max_requests=4, **kw):
    from nanoinfer_b200.config import load_config
    from nanoinfer_b200.engine import ModelRunner
    from nanoinfer_b200.weights import load_weights
    cfg = load_config(model_dir)
    num_pages = max(1, ru.max_live_tokens(steps, 64) // page)
    return ModelRunner(cfg, load_weights(model_dir, cfg), dtype=dtype, page_size=page, num_pages=num_pages,
                       max_requests=max_requests, **kw)


# ---- mechanisms alone ---------------------------------------------------------------------------------

@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rowwise_kernels(dtype):
    from nanoinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(5)
    tol = dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=1.6e-2, atol=1.6e-2)
    # embedding + sinusoid, odd width, positions far out
    table = torch.randn(50, 37, generator=g).to(dtype)
    tokens = torch.tensor([3, 49, 0, 7], dtype=torch.int32)
    pos = torch.tensor([0, 1, 511, 1290], dtype=torch.int32)
    i = torch.arange(19, dtype=torch.float64)
    inv = torch.pow(torch.tensor(10000.0, dtype=torch.float64), -2 * i / 37).float()
    out = torch.empty(4, 37, device=DEV)
    ops.embedding_sinusoid(tokens.to(DEV), pos.to(DEV), table.to(DEV), inv.to(DEV), out)
    want = table.double()[tokens.long()] + sinusoid(pos.tolist(), 37, torch.float64)
    torch.testing.assert_close(out.cpu().double(), want, rtol=0, atol=3e-4)     # FP32 angles at position 1290
    # PolyNorm, a width that is no multiple of the block
    z = (torch.randn(5, 203, generator=g) * 1.7).to(dtype)
    coef = torch.tensor([0.7, -0.4, 0.25, 0.1])
    act = torch.empty(5, 203, dtype=dtype, device=DEV)
    ops.polynorm(z.to(DEV), coef.to(DEV), 1e-5, act)
    zd = z.double()
    want = 0.7 * over_rms(zd, 1e-5) - 0.4 * over_rms(zd ** 2, 1e-5) + 0.25 * over_rms(zd ** 3, 1e-5) + 0.1
    torch.testing.assert_close(act.cpu().double(), want, **tol)
    # normed addition into the stream
    h = torch.randn(5, 203, generator=g)
    y = (torch.randn(5, 203, generator=g) * 3).to(dtype)
    wt = torch.rand(203, generator=g) + 0.5
    hd = h.clone().to(DEV)
    ops.add_normed(hd, y.to(DEV), wt.to(DEV), 1e-5)
    torch.testing.assert_close(hd.cpu().double(), h.double() + over_rms(y.double(), 1e-5) * wt.double(), rtol=2e-5, atol=2e-5)
    # gelu gate times a table row
    gate = torch.randn(4, 6, generator=g).to(dtype)
    tab = torch.randn(50, 30, generator=g).to(dtype)
    out = torch.empty(4, 6, dtype=dtype, device=DEV)
    ops.gelu_table_gate(gate.to(DEV), tokens.to(DEV), tab.to(DEV), 12, out)
    torch.testing.assert_close(out.cpu().double(), gelu_tanh(gate.double()) * tab.double()[tokens.long(), 12:18], **tol)


@pytest.mark.parametrize("G, H, D, V, taps", [(1, 2, 24, 40, 3), (2, 2, 160, 33, 1), (2, 6, 64, 48, 4), (1, 1, 8, 8, 6),
                                              (1, 1, 272, 16, 2), (1, 2, 520, 8, 2)])
def test_delta_kernels_alone(G, H, D, V, taps):
    """Two requests whose tokens arrive in three steps of unequal portions (long ones, which take the kernel's
    layout for long portions, and one shorter than the convolution's history), in slots that are not in order; the
    plain mixer gets the same inputs through projections that merely select columns."""
    from nanoinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(G + 10 * H + D)
    C, N = 2 * G * D + H * V, 2 * G * D + 2 * H * V + 2 * H
    lens = {"a": 43, "b": 9}
    inputs = {k: torch.randn(n, N, generator=g) for k, n in lens.items()}
    conv_w = torch.randn(C, taps, generator=g) * 0.6
    a_log, dt_bias = torch.randn(H, generator=g) - 2.0, torch.randn(H, generator=g)
    norm_w = torch.rand(V, generator=g) + 0.5
    state = torch.full((5, H * D * V + (taps - 1) * C), 7.0, device=DEV)
    slot = {"a": 3, "b": 1}
    for s in slot.values():
        state[s].zero_()
    got = {k: [] for k in lens}
    fed = {k: 0 for k in lens}
    for step in ({"a": 30, "b": 1}, {"b": 4, "a": 1}, {"a": 12, "b": 4}):
        ids = list(step)
        proj = torch.cat([inputs[k][fed[k]:fed[k] + step[k]] for k in ids]).to(DEV)
        n = proj.shape[0]
        cu = torch.tensor([0] + list(torch.tensor([step[k] for k in ids]).cumsum(0)), dtype=torch.int32, device=DEV)
        seq = torch.repeat_interleave(torch.arange(len(ids)), torch.tensor([step[k] for k in ids])).int().to(DEV)
        slots = torch.tensor([slot[k] for k in ids], dtype=torch.int32, device=DEV)
        qkv = torch.empty(n, C, device=DEV)
        gates = torch.empty(n, H, 2, device=DEV)
        ops.delta_prepare(proj, conv_w.to(DEV), a_log.to(DEV), dt_bias.to(DEV), state, seq, cu, slots, len(ids), G, H, D, V,
                          taps, qkv, gates)
        o = torch.empty(n, H * V, device=DEV)
        ops.delta_recurrence(qkv, gates, state, cu, slots, len(ids), G, H, D, V, o)
        y = torch.empty(n, H * V, device=DEV)
        ops.delta_gated_norm(o, proj, norm_w.to(DEV), 1e-5, G, H, D, V, y, state, cu, slots, len(ids), taps)
        at = 0
        for k in ids:
            got[k].append(y[at:at + step[k]].cpu())
            at += step[k]
            fed[k] += step[k]
    assert bool((state[0] == 7.0).all()) and bool((state[2] == 7.0).all()) and bool((state[4] == 7.0).all())
    eye = torch.eye(N, dtype=torch.float64)
    cols = {"q": (0, G * D), "k": (G * D, 2 * G * D), "v": (2 * G * D, C), "g": (C, C + H * V), "b": (C + H * V, C + H * V + H),
            "a": (C + H * V + H, N)}
    w = {k: eye[a:b] for k, (a, b) in cols.items()}
    w.update({"q.conv": conv_w[:G * D].double(), "k.conv": conv_w[G * D:2 * G * D].double(), "v.conv": conv_w[2 * G * D:].double(),
              "A_log": a_log.double(), "dt_bias": dt_bias.double(), "norm": norm_w.double(), "o": torch.eye(H * V, dtype=torch.float64)})
    m = {"heads": H, "kv_heads": G, "dim": D, "vdim": V, "conv": taps}
    for k in lens:
        want = delta_mixer(inputs[k].double(), w, m, 1e-5, delta_state(m, torch.float64))
        torch.testing.assert_close(torch.cat(got[k]).double(), want, rtol=2e-4, atol=2e-5)


@pytest.mark.parametrize("G, H, D, V, taps, fast", [(1, 1, 128, 128, 4, False), (2, 6, 64, 36, 4, False), (1, 2, 256, 68, 3, False),
                                                    (4, 4, 128, 32, 1, True), (1, 3, 64, 4, 6, True), (8, 160, 64, 32, 4, False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_delta_rule_by_blocks_of_four_tokens(G, H, D, V, taps, fast, dtype):
    """Portions of every length modulo four, shorter than the convolution's history too, requests without tokens beside them
    and slots out of order, in two steps: read-outs, states and histories against the kernel that walks the tokens one by one.
    ``fast``: decays that reach zero within a block (products of stretches only, no quotients)."""
    from nanoinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(G + 10 * H + D + V)
    C = 2 * G * D + H * V
    b_col = C + 4
    a_col, N = b_col + H, -(-(b_col + 2 * H) // 4) * 4
    conv_w, i32 = (torch.randn(C, taps, generator=g) * 0.6).to(DEV), dict(dtype=torch.int32, device=DEV)
    a_log = (torch.randn(H, generator=g) + (4.0 if fast else -2.0)).to(DEV)
    dt_bias = torch.randn(H, generator=g).to(DEV)
    states = [torch.zeros(9, H * D * V + (taps - 1) * C, device=DEV) for _ in range(2)]
    slots = torch.tensor([4, 0, 7, 2, 5, 8], **i32)
    for lens in ([9, 1, 0, 67, 2, 16], [3, 8, 5, 4, 130, 0]):
        n = sum(lens)
        proj = torch.randn(n, N, generator=g).to(DEV, dtype)
        cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), **i32)
        seq = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).int().to(DEV)
        o = [torch.empty(n, H * V, device=DEV) for _ in range(2)]
        qkv, gates = torch.empty(n, C, device=DEV), torch.empty(n, H, 2, device=DEV)
        ops.delta_prepare(proj, conv_w, a_log, dt_bias, states[0], seq, cu, slots, len(lens), G, H, D, V, taps, qkv, gates, b_col=b_col)
        ops.delta_recurrence(qkv, gates, states[0], cu, slots, len(lens), G, H, D, V, o[0])
        ops.delta_block_recurrence(proj, 0, b_col, a_col, conv_w, a_log, dt_bias, states[1], cu, slots, len(lens), G, H, D, V, taps, o[1])
        norm_w, gate = torch.ones(V, device=DEV), torch.ones(n, H * V, device=DEV)
        for k in range(2):
            ops.delta_gated_norm(o[k], proj, norm_w, 1e-5, G, H, D, V, torch.empty(n, H * V, dtype=dtype, device=DEV), states[k], cu, slots,
                                 len(lens), taps, gate=gate, gate_col=0)
        # sums of D terms in another order, carried along at most 130 tokens whose state neither rule lets grow
        scale = o[0].abs().max().item()
        torch.testing.assert_close(o[1], o[0], rtol=2e-5, atol=2e-5 * scale)
        assert torch.equal(states[0][:, H * D * V:], states[1][:, H * D * V:])                # the histories
        torch.testing.assert_close(states[1], states[0], rtol=2e-5, atol=2e-5 * states[0][:, :H * D * V].abs().max().item())
        states[1].copy_(states[0])
    assert bool((states[1][[1, 3, 6]] == 0).all())


@pytest.mark.parametrize("dtype, col0, extra, taken", [(torch.bfloat16, 4, 0, True), (torch.bfloat16, 1, 0, True), (torch.bfloat16, 0, 1, True),
                                                       (torch.float32, 4, 0, True), (torch.float32, 2, 0, False), (torch.float32, 0, 2, False)])
def test_delta_blocks_of_rows_that_start_anywhere(dtype, col0, extra, taken):
    """The rule that picks the blocks takes exactly the rows that the launcher takes: bfloat16 rows from any column on (a
    side of joined mixers starts where the other one ends), float32 rows on 16 bytes."""
    from nanoinfer_b200.kernels import ops
    G, H, D, V, taps, n = 1, 2, 64, 8, 4, 13
    C = 2 * G * D + H * V
    N = col0 + C + 2 * H + (-(col0 + C + 2 * H)) % 8 + extra
    g = torch.Generator().manual_seed(col0 + extra)
    proj, state = torch.randn(n, N, generator=g).to(DEV, dtype), torch.randn(1, H * D * V + (taps - 1) * C, generator=g).to(DEV)
    conv_w, a_log, dt_bias = (torch.randn(*s, generator=g).to(DEV) for s in ((C, taps), (H,), (H,)))
    i32 = dict(dtype=torch.int32, device=DEV)
    cu, slots, seq = torch.tensor([0, n], **i32), torch.zeros(1, **i32), torch.zeros(n, **i32)
    assert ops.delta_block_takes(proj, col0, state) == taken
    states, o = [state.clone(), state.clone()], [torch.empty(n, H * V, device=DEV) for _ in range(2)]
    block = lambda: ops.delta_block_recurrence(proj, col0, col0 + C, col0 + C + H, conv_w, a_log, dt_bias, states[1], cu, slots, 1, G, H, D, V,
                                               taps, o[1])
    if not taken:
        with pytest.raises(ops.KernelError):
            block()
        return
    block()
    qkv, gates = torch.empty(n, C, device=DEV), torch.empty(n, H, 2, device=DEV)
    ops.delta_prepare(proj, conv_w, a_log, dt_bias, states[0], seq, cu, slots, 1, G, H, D, V, taps, qkv, gates, col0=col0, b_col=col0 + C)
    ops.delta_recurrence(qkv, gates, states[0], cu, slots, 1, G, H, D, V, o[0])
    # sums of D terms in another order, along 13 tokens
    torch.testing.assert_close(o[1], o[0], rtol=2e-5, atol=2e-5 * o[0].abs().max().item())
    torch.testing.assert_close(states[1], states[0], rtol=2e-5, atol=2e-5 * states[0].abs().max().item())


def _one_layer(layer, width=64, vocab=120, side=None):
    raw = {"architecture": "Runevik", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "layers": [layer]}
    if side:
        raw["token_side"] = {"dim": side}
    return raw


def _far_token_matters(tmp_path, raw, tune, dtype, n=300, far=3, last=2):
    """A prompt whose last token (``last``) looks for token 2, which stands at position ``far`` and nowhere else;
    putting token 3 there instead must move the plain logits at the end by much, and the engine must follow
    both prompts."""
    from nanoinfer_b200.engine import StepEntry
    d = str(tmp_path / "m")
    tr.write_model(d, raw, 7, tune=tune)
    cfg, w = load_plain(d)
    plain = PlainRunevik(cfg, w)
    base = [5 + (i % 90) for i in range(n)]
    base[far], base[-1] = 2, last
    other = list(base)
    other[far] = 3
    want = {k: plain.run(t, plain.new_state())[0][-1].float() for k, t in (("same", base), ("other", other))}
    moved = (want["same"] - want["other"]).abs().max().item()
    assert moved > 0.1 * want["same"].abs().max().item(), "the test's weights do not make the far token count"
    steps = ru.whole({"same": base, "other": other})
    runner = _runner(d, dtype, steps, max_requests=2)
    for k, toks in (("same", base), ("other", other)):
        # most of the prompt at once, then portions that end at and just after page borders, then single tokens
        cuts = [0, 250, 256, 257, 272, 290] + list(range(291, n + 1))
        for a, b in zip(cuts, cuts[1:]):
            logits = runner.step([StepEntry(k, toks[a:b], [b - a - 1])])
        runner.end(k)
        ru.compare({(k, n - 1): logits[0].cpu()}, {k: {n - 1: want[k]}}, dtype, label=f"far token, {k}")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_latent_attention_finds_a_far_key(tmp_path, dtype):
    """Queries that look for their own token: q = s * W_uk W_dkv, so the score of a key is large where the key's
    token equals the query's; token identity dominates the embedding."""
    def tune(t):
        t["embed"].mul_(4.0)
        uk = t["l0.mix.uk"].float()
        t["l0.mix.q"].copy_((10.0 * uk @ t["l0.mix.dkv"].float()).to(t["l0.mix.q"].dtype))
        t["l0.mix.g"].zero_()
        t["l0.mix.o"].mul_(12.0)
    raw = _one_layer(tr.latent(2, 32, 24, 64, 0.5, 0))
    _far_token_matters(tmp_path, raw, tune, dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_delta_state_keeps_a_far_token(tmp_path, dtype):
    """Decays of nearly one.  Tokens 2 and 4 have a spike in one coordinate of their embedding that no other token
    has, token 3 in another; the key (and read-out query) projections turn each spike into a key of its own, so
    what token 2 wrote at position 3 stays untouched by the 295 tokens that follow and is read by token 4 at the
    end - unless token 3 stood there, which writes elsewhere."""
    def tune(t):
        e = t["embed"]
        e.mul_(4.0)
        e[:, 60] = 0
        e[:, 62] = 0
        e[2, 60] = e[4, 60] = e[3, 62] = 30.0
        k = t["l0.mix.k"]
        k[:, 60] = 0
        k[:, 62] = 0
        k[0] = 0
        k[1] = 0
        k[0, 60] = k[1, 62] = 1.0
        t["l0.mix.v"][:, 60] = 0
        t["l0.mix.v"][:, 62] = 0
        t["l0.mix.v"].mul_(5.0)
        t["l0.mix.q"].copy_(k)
        t["l0.mix.q.conv"].copy_(t["l0.mix.k.conv"])
        for name in ("l0.mix.q.conv", "l0.mix.k.conv", "l0.mix.v.conv"):
            t[name][:, :-1].mul_(0.1)                # mostly the current token
            t[name][:, -1] = t[name][:, -1].abs() + 0.5
        t["l0.mix.A_log"].fill_(-7.0)
        t["l0.mix.o"].mul_(6.0)
        t["l0.mix.g"].mul_(10.0)
    raw = _one_layer(tr.delta(2, 1, 64, 24, 3, 0))
    _far_token_matters(tmp_path, raw, tune, dtype, last=4)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_token_input_and_polynorm_alone(tmp_path, dtype):
    """One layer whose mixer is silenced (zero output projection): what is left is the feed-forward and the
    token input; with the feed-forward's output silenced too, only the token input."""
    for silence in (("l0.mix.o",), ("l0.mix.o", "l0.mlp.down")):
        def tune(t, silence=silence):
            for name in silence:
                t[name].zero_()
        raw = _one_layer(tr.delta(1, 1, 16, 16, 2, 72), width=48, side=12)
        d = str(tmp_path / ("m" + str(len(silence))))
        tr.write_model(d, raw, 9, tune=tune)
        cfg, w = load_plain(d)
        plain = PlainRunevik(cfg, w)
        reqs = {"a": random_tokens(120, 19, 1), "b": random_tokens(120, 2, 2)}
        want = {rid: plain.run(toks, plain.new_state())[0].float() for rid, toks in reqs.items()}
        steps = ru.ragged(reqs, sizes=(5, 2, 7))
        ru.compare(ru.run_trace(_runner(d, dtype, steps), steps), want, dtype, label="token input")


@pytest.mark.parametrize("heads, rank", [(17, 288), (20, 64), (3, 96), (18, 128)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_latent_ranks_and_head_counts(tmp_path, dtype, heads, rank):
    """Latents and head counts that the fast attention kernels take only in part or not at all - a latent wider
    than any of their heads (288), more than 16 heads over the shared row (the split-K kernel's limit), a rank of
    96 (prompt kernel only) - and a second layer that borrows the latent with other sizes."""
    raw = {"architecture": "Runevik", "vocab": 90, "width": 80, "norm": {"eps": 1e-6},
           "layers": [tr.latent(heads, 8, 8, rank, 0.35, 0), tr.latent(2, 24, 40, rank, 0.2, 48, kv_from=0)]}
    d = str(tmp_path / "m")
    tr.write_model(d, raw, 21)
    cfg, w = load_plain(d)
    plain = PlainRunevik(cfg, w)
    reqs = {"a": random_tokens(90, 45, 1), "b": random_tokens(90, 18, 2)}
    want = {rid: plain.run(toks, plain.new_state())[0].float() for rid, toks in reqs.items()}
    steps = ru.mixed(reqs, max_live=2)
    _compare(ru.run_trace(_runner(d, dtype, steps), steps), want, dtype, label=f"latent {heads} x {rank}")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_sizes_that_are_no_multiple_of_eight(tmp_path, dtype):
    """A width of 100, a latent of 40, keys of 20, values of 12, a token input of 6, a vocabulary of 131: no fast
    path takes these, and the rows of the caches and projections start on odd boundaries."""
    raw = {"architecture": "Runevik", "vocab": 131, "width": 100, "norm": {"eps": 1e-5}, "token_side": {"dim": 6},
           "layers": [tr.delta(3, 1, 20, 12, 3, 52), tr.latent(5, 12, 10, 40, 0.3, 36), tr.latent(2, 20, 14, 40, 0.25, 0, kv_from=1)]}
    d = str(tmp_path / "m")
    tr.write_model(d, raw, 33)
    cfg, w = load_plain(d)
    plain = PlainRunevik(cfg, w)
    reqs = {"a": random_tokens(131, 39, 1), "b": random_tokens(131, 21, 2), "c": random_tokens(131, 2, 3)}
    want = {rid: plain.run(toks, plain.new_state())[0].float() for rid, toks in reqs.items()}
    for cut in (ru.whole, lambda r: ru.mixed(r, max_live=3)):
        steps = cut(reqs)
        _compare(ru.run_trace(_runner(d, dtype, steps), steps), want, dtype, label="odd sizes")


# ---- whole models, cut in four ways ---------------------------------------------------------------------

@pytest.mark.parametrize("cut", list(CUTS))
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("key", list(RAW))
def test_replay_matches_plain(models, key, dtype, cut):
    d, cfg, reqs, want = models[key]
    steps = CUTS[cut](reqs)
    runner = _runner(d, dtype, steps)
    got = ru.run_trace(runner, steps)
    assert len(got) == sum(len(t) for t in reqs.values())
    _compare(got, want, dtype, label=f"{key} {cut}", sensitivity=SENSITIVITY[key])
    runner.cache.check_consistency()
    assert runner.cache.num_free_slots == 4


@pytest.mark.parametrize("key", list(RAW))
def test_float32_does_not_depend_on_the_cut(models, key):
    """In 32-bit every cut gives the same bits: portions, batches, pages and slots only move data."""
    d, cfg, reqs, want = models[key]
    ref = None
    for cut in CUTS:
        steps = CUTS[cut](reqs)
        got = ru.run_trace(_runner(d, "float32", steps), steps)
        if ref is None:
            ref = got
        else:
            for k in ref:
                assert torch.equal(ref[k], got[k]), f"{key}: {cut} differs from whole at {k}"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_long_decoding_with_replayed_graphs(models, dtype):
    """Most of a request token by token (the steps are captured and replayed from the third on), a second request
    decoding beside it from the middle on."""
    d, cfg, reqs, want = models["r2"]
    reqs = {k: reqs[k] for k in ("q3", "q5")}
    steps = ru.tail_by_token({"q3": reqs["q3"]}, tail=140)
    join = ru.tail_by_token({"q5": reqs["q5"]}, tail=60)
    for i, st in enumerate(join):                       # q5 runs beside q3's single tokens
        steps[30 + i]["entries"] += st["entries"]
        steps[30 + i]["end"] += st["end"]
    runner = _runner(d, dtype, steps)
    _compare(ru.run_trace(runner, steps), want, dtype, label="long decoding", sensitivity=SENSITIVITY["r2"])
    assert runner._graphs, "no step of single tokens was captured"


def test_greedy_generation_through_the_engine(models):
    """Engine.generate (scheduler, chunked prompts, sampling kernels) against greedy decoding of the plain model."""
    from nanoinfer_b200 import Engine, SamplingParams
    d, cfg, reqs, want = models["r1"]
    raw_cfg, w = load_plain(d)
    plain = PlainRunevik(raw_cfg, w)
    prompts = [reqs["q2"], reqs["q3"][:20], reqs["q1"]]
    engine = Engine.from_model_dir(d, dtype="float32", block_size=16, num_cache_blocks=64, max_batch_size=4,
                                   max_sequences=4, prefill_chunk_size=12)
    out = engine.generate(prompts, max_new_tokens=12, sampling_params=SamplingParams.greedy())
    for prompt, got in zip(prompts, out):
        st = plain.new_state()
        logits = plain.run(prompt, st)[0][-1]
        for t in got:
            top2 = torch.topk(logits, 2).values
            if int(torch.argmax(logits)) != t:
                assert (top2[0] - logits[t]).item() < 1e-4, "the engine chose a token that the plain model ranks lower"
            logits = plain.run([t], st)[0][-1]
        assert len(got) == 12
