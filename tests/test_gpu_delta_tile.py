"""The gated delta rule sixteen tokens at a time against the kernel that walks the tokens one by one and against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(G, H, V, taps, lens, fast, seed, dtype=torch.float32, col0=0):
    g = torch.Generator().manual_seed(seed)
    C = 2 * G * 128 + H * V
    b_col = col0 + C + 4
    a_col = b_col + H
    N = -(-(b_col + 2 * H) // 4) * 4
    i32 = dict(dtype=torch.int32, device=DEV)
    return dict(G=G, H=H, V=V, taps=taps, C=C, b_col=b_col, a_col=a_col, col0=col0, n=sum(lens), n_seqs=len(lens),
                proj=torch.randn(sum(lens), N, generator=g).to(DEV, dtype), conv_w=(torch.randn(C, taps, generator=g) * 0.6).to(DEV),
                a_log=(torch.randn(H, generator=g) + fast).to(DEV), dt_bias=torch.randn(H, generator=g).to(DEV),
                cu=torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), **i32), slots=torch.randperm(len(lens) + 3, generator=g)[:len(lens)].int().to(DEV),
                seq=torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).int().to(DEV),
                state=torch.randn(len(lens) + 3, H * 128 * V + (taps - 1) * C, generator=g).to(DEV) * 0.2)


def _tiles(ops, x, tiles=True):
    state, out = x["state"].clone(), torch.full((x["n"], x["H"] * x["V"]), float("nan"), device=DEV)
    ops.delta_block_recurrence(x["proj"], x["col0"], x["b_col"], x["a_col"], x["conv_w"], x["a_log"], x["dt_bias"], state, x["cu"], x["slots"],
                               x["n_seqs"], x["G"], x["H"], 128, x["V"], x["taps"], out, tiles=tiles)
    return out, state


def _tokens(ops, x):
    state, out = x["state"].clone(), torch.empty(x["n"], x["H"] * x["V"], device=DEV)
    qkv, gates = torch.empty(x["n"], x["C"], device=DEV), torch.empty(x["n"], x["H"], 2, device=DEV)
    ops.delta_prepare(x["proj"], x["conv_w"], x["a_log"], x["dt_bias"], state, x["seq"], x["cu"], x["slots"], x["n_seqs"], x["G"], x["H"], 128,
                      x["V"], x["taps"], qkv, gates, col0=x["col0"], b_col=x["b_col"])
    ops.delta_recurrence(qkv, gates, state, x["cu"], x["slots"], x["n_seqs"], x["G"], x["H"], 128, x["V"], out)
    return out, state, qkv, gates


@pytest.mark.parametrize("G, H, V, taps, fast", [(1, 1, 128, 4, -2.0), (2, 6, 48, 4, -2.0), (4, 4, 32, 1, 4.0), (1, 3, 16, 6, 4.0), (2, 2, 80, 3, -6.0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_portions_of_every_length(G, H, V, taps, fast, dtype):
    """Portions around multiples of sixteen, shorter than the convolution's history, none at all, slots out of order; decays
    that reach zero within a tile and that hardly forget."""
    from nanoinfer_b200.kernels import ops
    x = _inputs(G, H, V, taps, [17, 1, 0, 67, 2, 16, 31, 33, 130, 15], fast, G + 10 * H + V, dtype)
    out, state = _tiles(ops, x)
    want, want_state, _, _ = _tokens(ops, x)
    # sums of 128 terms in another order, carried along at most 130 tokens whose state neither rule lets grow
    torch.testing.assert_close(out, want, rtol=2e-5, atol=2e-5 * want.abs().max().item())
    torch.testing.assert_close(state, want_state, rtol=2e-5, atol=2e-5 * want_state.abs().max().item())
    others = torch.ones(state.shape[0], dtype=torch.bool)
    others[x["slots"].long().cpu()] = False
    assert torch.equal(state[others], x["state"][others])


def _in_64_bits(x):
    G, H, V, taps, C, cu = x["G"], x["H"], x["V"], x["taps"], x["C"], x["cu"].tolist()
    proj, want, ends = x["proj"].double(), [], []
    decay = torch.exp(-torch.exp(x["a_log"].double()) * torch.nn.functional.softplus(proj[:, x["a_col"]:x["a_col"] + H] + x["dt_bias"].double()))
    beta = torch.sigmoid(proj[:, x["b_col"]:x["b_col"] + H])
    for r in range(x["n_seqs"]):
        kept = x["state"][x["slots"][r].long()].double()
        s, L = kept[:H * 128 * V].view(H, 128, V).clone(), cu[r + 1] - cu[r]
        rows = torch.cat([kept[H * 128 * V:].view(taps - 1, C), proj[cu[r]:cu[r + 1], x["col0"]:x["col0"] + C]])
        y = torch.nn.functional.silu(sum(rows[i:i + L] * x["conv_w"][:, i].double() for i in range(taps)))
        q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (y[:, :G * 128].view(L, G, 128), y[:, G * 128:2 * G * 128].view(L, G, 128)))
        q, k, v = q.repeat_interleave(H // G, 1) * 128 ** -0.5, k.repeat_interleave(H // G, 1), y[:, 2 * G * 128:].view(L, H, V)
        for t in range(L):
            s = s * decay[cu[r] + t][:, None, None]
            s = s + k[t][:, :, None] * (beta[cu[r] + t][:, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], s)))[:, None, :]
            want.append(torch.einsum("hd,hdv->hv", q[t], s).reshape(-1))
        ends.append(s.reshape(-1))
    return torch.stack(want), torch.stack(ends)


@pytest.mark.parametrize("lens", [[200, 130, 70], [1100]])
@pytest.mark.parametrize("fast", [-6.0, -4.0, -1.0, 2.0, 4.0])
def test_errors_against_64_bits_stay_where_they_were(fast, lens):
    """Read-outs and states no further from 64 bits than in blocks of four, in the mean over four inputs: decays near one, whose own
    errors add up along a long portion, to decays of a token or two, where every product's rounding shows."""
    from nanoinfer_b200.kernels import ops
    sums = {True: [0.0, 0.0], False: [0.0, 0.0]}
    for seed in range(4):
        x = _inputs(4, 4, 64, 4, lens, fast, 100 + seed)
        want, ends = _in_64_bits(x)
        for tiles, at in sums.items():
            out, state = _tiles(ops, x, tiles)
            end = state[x["slots"].long(), :4 * 128 * 64].double()
            at[0] += ((out - want).norm() / want.norm()).item()
            at[1] += ((end - ends).norm() / ends.norm()).item()
    assert all(a <= b for a, b in zip(sums[True], sums[False])), sums


def test_refused_and_chosen():
    from nanoinfer_b200.kernels import ops
    x = _inputs(1, 1, 20, 4, [200], -2.0, 6)
    with pytest.raises(ops.KernelError):
        _tiles(ops, x)                                       # value heads of 20
    out, _ = _tiles(ops, x, tiles=None)                      # ... go in blocks of four
    torch.testing.assert_close(out, _tokens(ops, x)[0], rtol=2e-5, atol=2e-5 * out.abs().max().item())
    x = _inputs(1, 2, 32, 4, [200], -2.0, 7, torch.bfloat16, col0=3)
    assert ops.delta_tile_pays(200, 1, 128, 32)
    assert torch.equal(_tiles(ops, x)[0], _tiles(ops, x, tiles=None)[0])


def test_a_buffer_of_the_caller_s_gives_the_same_bits():
    from nanoinfer_b200.kernels import ops
    x = _inputs(2, 4, 48, 4, [33, 180, 7], -2.0, 8)
    want, want_state = _tiles(ops, x)
    need = sum(ops.delta_tile_bytes(x["n"], x["n_seqs"], 2, 4, 48))
    buf = torch.full((need + 64,), 255, dtype=torch.uint8, device=DEV)       # (NaN wherever it is read before it is written)
    state, out = x["state"].clone(), torch.empty_like(want)
    args = (x["proj"], 0, x["b_col"], x["a_col"], x["conv_w"], x["a_log"], x["dt_bias"], state, x["cu"], x["slots"], x["n_seqs"], 2, 4, 128, 48, 4, out)
    with pytest.raises(ops.KernelError, match="too small"):
        ops.delta_block_recurrence(*args, tiles=True, buf=buf[:need - 1])
    ops.delta_block_recurrence(*args, tiles=True, buf=buf)
    assert torch.equal(out, want) and torch.equal(state, want_state) and (buf[need:] == 255).all()


def test_layers_and_captured_steps_share_one_buffer():
    """The part takes its scratch from the runtime: a second call, or another layer's, allocates none."""
    import types

    from nanoinfer_b200.kernels import ops
    from nanoinfer_b200.parts.recurrent import GatedDeltaRule
    x = _inputs(2, 2, 32, 4, [200, 60], -2.0, 9, torch.bfloat16)
    asked = []
    rt = types.SimpleNamespace(dtype=torch.bfloat16, empty=lambda *s, dtype=None: torch.zeros(s, device=DEV, dtype=dtype or torch.bfloat16),
                               workspace=lambda name, n, dtype, zero=False: asked.append((name, n)) or torch.empty(n, dtype=dtype, device=DEV))
    part = object.__new__(GatedDeltaRule)
    part.__dict__.update(rt=rt, G=2, H=2, D=128, V=32, taps=4, channels=x["C"], b_col=x["b_col"], gate_col=0, wants_f32_tokens=False, w_thin=None,
                         channel=False, chunked=False, in_blocks=True, thin_gate=False, conv_w=x["conv_w"], a_log=x["a_log"], dt_bias=x["dt_bias"],
                         norm_w=torch.ones(32, device=DEV), eps=1e-6, output_scale=1.0)
    ctx = types.SimpleNamespace(max_q_len=200, n_seqs=2, cu_q=x["cu"], slots=x["slots"], seq_of_token=x["seq"])
    out = torch.empty(260, 64, dtype=torch.bfloat16, device=DEV)
    for _ in range(2):
        part.between(x["proj"], 0, ctx, types.SimpleNamespace(state=x["state"].clone()), out)
    assert asked == [("delta_tiles", sum(ops.delta_tile_bytes(260, 2, 2, 2, 32)))] * 2


@pytest.mark.parametrize("poison", [float("inf"), float("nan")])
@pytest.mark.parametrize("what", ["value", "key", "query", "beta", "decay"])
def test_what_is_not_finite_stays_with_its_own_and_later_tokens(poison, what):
    """An infinity or a NaN in the middle of a tile: tokens before it, other requests and (a value) other columns as if it were not there."""
    from nanoinfer_b200.kernels import ops
    x = _inputs(2, 2, 32, 4, [45, 40], -2.0, 11)
    clean, clean_state = _tiles(ops, x)
    column = {"value": 2 * 2 * 128 + 32 + 5, "key": 2 * 128 + 128 + 7, "query": 128 + 3, "beta": x["b_col"] + 1, "decay": x["a_col"] + 1}[what]
    x["proj"][22, column] = poison                            # head 1 of request 0
    out, state = _tiles(ops, x)
    hit = torch.zeros_like(clean, dtype=torch.bool)
    hit[22:45, 32 + 5 if what == "value" else slice(32, 64)] = True
    torch.testing.assert_close(out[~hit], clean[~hit], rtol=1e-6, atol=1e-6 * clean.abs().max().item())
    want, want_state, _, _ = _tokens(ops, x)
    keep = torch.isfinite(want)
    assert torch.equal(torch.isfinite(out)[~hit], keep[~hit]) and not torch.isfinite(out[~keep]).any()
    torch.testing.assert_close(state[x["slots"][1].long()], clean_state[x["slots"][1].long()], rtol=0, atol=0)
