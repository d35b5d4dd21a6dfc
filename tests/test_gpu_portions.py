"""Prompt-side kernels at the edges of their tiles against the plain recurrences / sums in float64."""
import pytest
import torch

from llmss_b200 import ops
from llmss_b200.engine.batch import BatchInput

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64


def _batch(lens, ctxs, slots):
    cu = torch.tensor([0] + list(lens)).cumsum(0).to(torch.int32)
    i32 = dict(dtype=torch.int32, device="cuda")
    z = torch.zeros(1, **i32)
    return BatchInput(tokens=z, positions=z, slot_mapping=z, block_tables=z.view(1, 1), seq_lens=torch.tensor([a + b for a, b in zip(lens, ctxs)], **i32),
                      cu_q=cu.cuda(), last_idx=z, num_seqs=len(lens), max_q=max(lens), max_kv=1, is_decode=False, is_fresh_prefill=False,
                      state_slots=torch.tensor(slots, **i32))


def _rel(got, want):
    return float((got.double().cpu() - want).norm() / want.norm().clamp_min(1e-30))


@pytest.mark.parametrize("dk,dv,heads,qk_heads,unit", [(128, 128, 2, 1, True), (64, 64, 2, 2, True), (24, 16, 2, 1, False), (8, 3, 3, 3, True),
                                                       (100, 70, 2, 2, True), (200, 40, 1, 1, False), (300, 10, 1, 1, True)])
@pytest.mark.parametrize("copies", [1, 40])
def test_delta_portions(dk, dv, heads, qk_heads, unit, copies):
    """Portions around the 16-token stages, states carried over, key sizes that take 1 to 16 lanes to a column pair; ``copies`` = 40: more
    blocks than the GPU holds at once, over as many state slots.  Bound: 32-bit sums, 3e-6 of the norm."""
    torch.manual_seed(dk + dv)
    lens, ctxs = [16, 1, 33, 47][:4 if copies == 1 else 2] * copies, [0, 3, 8, 0][:4 if copies == 1 else 2] * copies
    slots, T = list(range(len(lens))), sum(lens)
    q, k, v = (torch.randn(T, n, device="cuda") for n in (qk_heads * dk, qk_heads * dk, heads * dv))
    if not unit:        # keys of norm 1 keep the rule stable
        k = torch.nn.functional.normalize(k.view(T, qk_heads, dk), dim=-1).reshape(T, -1)
    g, b = -torch.rand(T, heads, device="cuda") * 0.3, torch.randn(T, heads, device="cuda")
    state = torch.randn(len(lens), heads, dk, dv, device="cuda") * 0.1
    S0 = state.reshape(len(lens), heads, dv, dk).transpose(2, 3).double().cpu()
    rep = heads // qk_heads
    qf, kf = (x.double().cpu().view(T, qk_heads, dk) for x in (q, k))
    if unit:
        qf, kf = (x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6) for x in (qf, kf))
    qf, kf, vf = (qf * 0.25).repeat_interleave(rep, 1), kf.repeat_interleave(rep, 1), v.double().cpu().view(T, heads, dv)
    a, beta = torch.exp(g.double().cpu()), torch.sigmoid(b.double().cpu())
    want, at, ends = torch.zeros_like(vf), 0, []
    for i, n in enumerate(lens):
        S = S0[i].clone() if ctxs[i] else torch.zeros(heads, dk, dv, dtype=F64)
        for t in range(at, at + n):
            S = S * a[t][:, None, None]
            u = beta[t][:, None] * (vf[t] - torch.einsum("hkv,hk->hv", S, kf[t]))
            S = S + kf[t][:, :, None] * u[:, None, :]
            want[t] = torch.einsum("hkv,hk->hv", S, qf[t])
        ends.append(S)
        at += n
    got = ops.delta_scan(q, k, v, g, b, _batch(lens, ctxs, slots), state, heads, qk_heads, dk, dv, unit_eps=1e-6 if unit else None, q_scale=0.25,
                         beta_sigmoid=True)
    assert _rel(got, want.reshape(T, -1)) < 3e-6
    assert _rel(state.reshape(len(lens), heads, dv, dk).transpose(2, 3), torch.stack(ends)) < 3e-6


def _delta64(q, k, v, g, beta, S0, lens, ctxs, heads, qk_heads, dk, dv, unit):
    rep, T = heads // qk_heads, sum(lens)
    qf, kf = (x.double().cpu().reshape(T, qk_heads, dk) for x in (q, k))
    if unit:
        qf, kf = (x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6) for x in (qf, kf))
    qf, kf, vf = (qf * 0.25).repeat_interleave(rep, 1), kf.repeat_interleave(rep, 1), v.double().cpu().reshape(T, heads, dv)
    a, beta = torch.exp(g.double().cpu()), torch.sigmoid(beta.double().cpu())
    out, ends, at = torch.zeros_like(vf), [], 0
    for i, n in enumerate(lens):
        S = S0[i].clone() if ctxs[i] else torch.zeros(heads, dk, dv, dtype=F64)
        for t in range(at, at + n):
            S = S * a[t][:, None, None]
            u = beta[t][:, None] * (vf[t] - torch.einsum("hkv,hk->hv", S, kf[t]))
            S = S + kf[t][:, :, None] * u[:, None, :]
            out[t] = torch.einsum("hkv,hk->hv", S, qf[t])
        ends.append(S)
        at += n
    return out, torch.stack(ends)


def _delta_inputs(lens, heads, qk_heads, dk, dv, unit, wide=0):
    T = sum(lens)
    rows = [torch.randn(T, n + wide, device="cuda")[:, wide:] for n in (qk_heads * dk, qk_heads * dk, heads * dv)]
    if not unit:        # keys of norm 1 keep the rule stable
        rows[1] = torch.nn.functional.normalize(rows[1].reshape(T, qk_heads, dk), dim=-1).reshape(T, -1)
    return rows, torch.randn(T, heads, device="cuda"), torch.randn(len(lens), heads, dk, dv, device="cuda") * 0.1


@pytest.mark.parametrize("dk,dv,heads,qk_heads,unit", [(128, 128, 2, 1, True), (128, 128, 3, 3, False), (64, 48, 2, 2, True), (100, 200, 6, 2, True), (4, 3, 1, 1, True)])
@pytest.mark.parametrize("decay", ["mild", "slow", "strong", "one", "above one"])
def test_delta_over_chunks(dk, dv, heads, qk_heads, unit, decay, monkeypatch):
    """Portions around the 32-token chunks, shorter ones beside them, states carried over, rows of wider tensors, key heads of one and more value
    heads; decays that leave nothing of a chunk's start, decays of exactly one, and growing ones (token by token inside their chunks).  Bound:
    32-bit sums, 1e-6 of the norm (growth over 100 tokens multiplies it)."""
    from llmss_b200.ops import cuda_impl as cu

    monkeypatch.setattr(cu, "_delta_over_chunks", lambda *a: True)
    torch.manual_seed(dk + dv)
    lens, ctxs = [32, 7, 100, 33, 64, 31], [0, 5, 8, 0, 3, 2]
    (q, k, v), b, S0 = _delta_inputs(lens, heads, qk_heads, dk, dv, unit, wide=4)
    u = torch.rand(sum(lens), heads, device="cuda")
    g = {"mild": -0.3 * u, "slow": -0.01 * u, "strong": -3.0 - 9.0 * u, "one": 0.0 * u, "above one": 0.6 * u - 0.25}[decay]
    state = S0.transpose(2, 3).contiguous().view(len(lens), heads, dk, dv)
    want, ends = _delta64(q, k, v, g, b, S0.double().cpu(), lens, ctxs, heads, qk_heads, dk, dv, unit)
    got = ops.delta_scan(q, k, v, g, b, _batch(lens, ctxs, range(len(lens))), state, heads, qk_heads, dk, dv, unit_eps=1e-6 if unit else None,
                         q_scale=0.25, beta_sigmoid=True)
    bound = 1e-5 if decay == "above one" else 1e-6
    assert _rel(got, want.reshape(sum(lens), -1)) < bound
    assert _rel(state.reshape(len(lens), heads, dv, dk).transpose(2, 3), ends) < bound


@pytest.mark.parametrize("n,max_q", [(1, 1), (7, 7), (31, 31), (31, 64), (32, 32), (7, 0), (100, 64), (100, 40)])
def test_delta_over_chunks_of_one_sequence(n, max_q):
    """The C entry, one sequence of any length: a short one runs token by token, and ``max_q`` is a hint on the lengths: tokens
    beyond it run token by token."""
    from llmss_b200.ops import _lib, cuda_impl as cu

    torch.manual_seed(n)
    heads, d = 2, 64
    (q, k, v), b, S0 = _delta_inputs([n], heads, heads, d, d, True)
    g, batch = -0.3 * torch.rand(n, heads, device="cuda"), _batch([n], [3], [0])
    state, out = S0.transpose(2, 3).contiguous(), torch.full((n, heads * d), float("nan"), device="cuda")
    want, ends = _delta64(q, k, v, g, b, S0.double().cpu(), [n], [3], heads, heads, d, d, True)
    lib, p = _lib.load(), cu._ptr
    scratch = torch.empty(lib.llmss_delta_scan_chunked_bytes(n, 1, heads), dtype=torch.uint8, device="cuda")
    _lib.check(lib.llmss_delta_scan_chunked(p(q), q.stride(0), p(k), k.stride(0), p(v), v.stride(0), p(g), heads, p(b), heads, p(out), p(state), p(batch.cu_q),
                                            p(batch.seq_lens), p(batch.state_slots), 1, max_q, heads, heads, d, d, 1e-6, 0.25, 1, p(scratch), cu._stream()), "chunked")
    assert _rel(out, want.reshape(n, -1)) < 1e-6 and _rel(state.transpose(2, 3), ends) < 1e-6


@pytest.mark.parametrize("dk,dv,heads,qk_heads", [(128, 128, 4, 2), (20, 300, 2, 2), (64, 70, 2, 1)])
@pytest.mark.parametrize("tokens", [[0], [40, 99], [32 + 107, 99 + 3], [107 + 63, 107 + 64 + 32]])
def test_delta_over_chunks_until_a_chunk_that_grows(dk, dv, heads, qk_heads, tokens, monkeypatch):
    """One token with a growing decay in the first, a middle or the last chunk of some sequences and one head: what is left of those runs token by
    token behind, from the state in front of the chunk, and nothing else changes.  Bound: 32-bit sums, 1e-6 of the norm."""
    from llmss_b200.ops import cuda_impl as cu

    monkeypatch.setattr(cu, "_delta_over_chunks", lambda *a: True)
    torch.manual_seed(dk + dv)
    lens, ctxs, slots = [100, 7, 64, 33], [0, 5, 8, 2], [2, 0, 3, 1]
    (q, k, v), b, S0 = _delta_inputs(lens, heads, qk_heads, dk, dv, True)
    g = -0.3 * torch.rand(sum(lens), heads, device="cuda")
    g[tokens, 1] = 0.3
    state = torch.empty(len(lens), heads, dk, dv, device="cuda")
    state.view(len(lens), heads, dv, dk)[slots] = S0.transpose(2, 3)
    want, ends = _delta64(q, k, v, g, b, S0.double().cpu(), lens, ctxs, heads, qk_heads, dk, dv, True)
    got = ops.delta_scan(q, k, v, g, b, _batch(lens, ctxs, slots), state, heads, qk_heads, dk, dv, unit_eps=1e-6, q_scale=0.25, beta_sigmoid=True)
    assert _rel(got, want.reshape(sum(lens), -1)) < 1e-6
    assert _rel(state.view(len(lens), heads, dv, dk)[slots].transpose(2, 3), ends) < 1e-6


def test_delta_over_chunks_costs_no_more_where_it_cannot_be_used(monkeypatch):
    """Decays that grow in every chunk: one pass over the portions token by token and what the chunks' launches take to notice (token by token in
    the chunks' own kernel it was 5.8 times as long)."""
    from llmss_b200.ops import cuda_impl as cu

    torch.manual_seed(1)
    lens, heads, d = [512] * 4, 8, 128
    (q, k, v), b, S0 = _delta_inputs(lens, heads, 4, d, d, True)
    g, state, batch = 0.26 + 0.04 * torch.rand(sum(lens), heads, device="cuda"), S0, _batch(lens, [0] * 4, range(4))

    def best(form):
        monkeypatch.setattr(cu, "_delta_over_chunks", lambda *a: form)
        times = []
        for _ in range(8):
            at = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            at[0].record()
            ops.delta_scan(q, k, v, g, b, batch, state, heads, 4, d, d, unit_eps=1e-6, q_scale=0.25, beta_sigmoid=True)
            at[1].record()
            torch.cuda.synchronize()
            times.append(at[0].elapsed_time(at[1]))
        return min(times[2:])

    assert best(True) < 1.6 * best(False)


def test_delta_over_chunks_in_odd_batches(monkeypatch):
    """An empty sequence, one without a slot, slots in another order than the batch, scratch that holds other bytes; then the same call captured and
    replayed from the same state, and with rows off the 16-byte lines (token by token).  Bound: 32-bit sums, 1e-6 of the norm."""
    from llmss_b200.ops import cuda_impl as cu

    monkeypatch.setattr(cu, "_delta_over_chunks", lambda *a: True)
    torch.manual_seed(6)
    lens, ctxs, slots, heads, qk_heads, d = [64, 0, 40, 5, 97], [0, 4, 3, 2, 6], [3, 1, -1, 0, 5], 4, 2, 128
    T, rows = sum(lens), slice(64, 104)
    (q, k, v), b, S0 = _delta_inputs(lens, heads, qk_heads, d, d, True)
    g, batch = -0.3 * torch.rand(T, heads, device="cuda"), _batch(lens, ctxs, slots)
    start = torch.randn(6, heads, d, d, device="cuda")
    live = [i for i in range(len(lens)) if slots[i] >= 0 and lens[i]]
    start[[slots[i] for i in live]] = S0[live].transpose(2, 3)
    want, ends = _delta64(q, k, v, g, b, S0.double().cpu(), lens, ctxs, heads, qk_heads, d, d, True)

    def check(got, state):
        got = torch.cat([got[:rows.start], got[rows.stop:]])
        assert _rel(got, torch.cat([want[:rows.start], want[rows.stop:]]).reshape(got.shape)) < 1e-6
        assert _rel(state[[slots[i] for i in live]].transpose(2, 3), ends[live]) < 1e-6
        assert torch.equal(state[[1, 2, 4]], start[[1, 2, 4]])          # nobody's, an empty sequence's

    def call(q, k, state):
        return ops.delta_scan(q, k, v, g, b, batch, state, heads, qk_heads, d, d, unit_eps=1e-6, q_scale=0.25, beta_sigmoid=True)

    dirty = torch.full((1 << 20,), 255, dtype=torch.uint8, device="cuda")
    del dirty
    state = start.clone()
    eager = call(q, k, state)
    check(eager, state)

    held, graph = start.clone(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call(q, k, held)
    for _ in range(2):
        held.copy_(start)
        graph.replay()
        assert torch.equal(held, state) and torch.equal(out[:rows.start], eager[:rows.start]) and torch.equal(out[rows.stop:], eager[rows.stop:])

    off = [torch.empty(T, x.shape[1] + 1, device="cuda")[:, 1:].copy_(x) for x in (q, k)]
    state = start.clone()
    check(call(*off, state), state)


def _delta_worst(got, want, dims):
    """Largest error of a part (a token of a head, a column, ..) over the norm of that part."""
    return float(((got.double().cpu() - want).norm(dim=dims) / want.norm(dim=dims).clamp_min(1e-300)).max())


def test_delta_over_chunks_channels_of_unequal_size(monkeypatch):
    """Key channels between 2^-6 and 2^6, queries the other way round: small entries of the state meet large ones of the queries.  Bound: 2^-24 a term,
    64 of them: 4e-6 of each token and head (token by token 5e-7; a state of two 16-bit parts: 8e-5)."""
    from llmss_b200.ops import cuda_impl as cu

    monkeypatch.setattr(cu, "_delta_over_chunks", lambda *a: True)
    torch.manual_seed(3)
    n, heads, d = 160, 2, 128
    (q, k, v), b, S0 = _delta_inputs([n], heads, heads, d, d, True)
    size = torch.exp2(torch.rand(d, device="cuda") * 12 - 6)
    k.view(n, heads, d).mul_(size), q.view(n, heads, d).div_(size)
    g, state = -0.3 * torch.rand(n, heads, device="cuda"), S0.transpose(2, 3).contiguous()
    want, ends = _delta64(q, k, v, g, b, S0.double().cpu(), [n], [0], heads, heads, d, d, True)
    got = ops.delta_scan(q, k, v, g, b, _batch([n], [0], [0]), state, heads, heads, d, d, unit_eps=1e-6, q_scale=0.25, beta_sigmoid=True).view(n, heads, d)
    assert _delta_worst(got, want, 2) < 4e-6
    assert _delta_worst(state.transpose(2, 3), ends, 3) < 4e-6          # each key row of the state


@pytest.mark.parametrize("what", ["1e3", "1e6", "1e12", "1e29", "early 1e12", "forgotten 1e6", "unequal tokens", "forgetful", "sparse keys", "small first token"])
def test_delta_over_chunks_wide_numbers(what, monkeypatch):
    """Numbers of very different size in one chunk and column: a large value takes nothing from the tokens in front of it, from other columns, or from
    tokens behind a decay that has forgotten it; tokens of 2^-12 to 2^12, also where each stands alone (strong decays; keys with one channel each).  Bound: 2^-24 a
    term, 32 of them: 2e-6 of every token's own norm, tokens behind a value that the rule itself cancels left out."""
    from llmss_b200.ops import cuda_impl as cu

    monkeypatch.setattr(cu, "_delta_over_chunks", lambda *a: True)
    torch.manual_seed(4)
    n, heads, d = 160, 2, 128
    (q, k, v), b, S0 = _delta_inputs([n], heads, heads, d, d, True)
    u, at, ctx, last = torch.rand(n, heads, device="cuda"), 77, 3, n
    g, V = -0.3 * u, v.view(n, heads, d)
    if what[-1].isdigit():
        at = 66 if "early" in what else at
        V[at, 1, 7] = float(what.split()[-1])
        if "forgotten" in what:
            g = torch.where(u < 0.2, -40.0, g)
        else:
            last = at
    elif what == "small first token":
        ctx, V[0] = 0, V[0] * 2.0 ** -20
    else:
        V.mul_(torch.exp2(torch.rand(n, 1, 1, device="cuda") * 24 - 12))
    if what == "forgetful":
        g = -3.0 - 9.0 * u
    if what == "sparse keys":
        i = torch.randint(0, d, (n, heads, 1), device="cuda")
        k.zero_().view(n, heads, d).scatter_(2, i, 1.0)
        q.zero_().view(n, heads, d).scatter_(2, i.roll(3, 0), 1.0)
    state = S0.transpose(2, 3).contiguous()
    want, ends = _delta64(q, k, v, g, b, S0.double().cpu(), [n], [ctx], heads, heads, d, d, True)
    got = ops.delta_scan(q, k, v, g, b, _batch([n], [ctx], [0]), state, heads, heads, d, d, unit_eps=1e-6, q_scale=0.25, beta_sigmoid=True).view(n, heads, d)
    keep = want[:last].norm(dim=(1, 2)) > 0
    assert _delta_worst(got[:last][keep.cuda()], want[:last][keep], (1, 2)) < 2e-6
    others = [i for i in range(d) if i != 7]
    assert _delta_worst(got[..., others], want[..., others], 0) < 1e-6              # each other column over all tokens
    assert _delta_worst(state.transpose(2, 3)[..., others], ends[..., others], 2) < 1e-6


@pytest.mark.parametrize("decay,stays", [("mild", True), ("slow", True), ("strong", True), ("resets", True), ("strong, unequal tokens", False), ("growing", False)])
def test_delta_over_chunks_keeps_ordinary_inputs(decay, stays):
    """The record of a sequence's first chunk says how many tokens went over chunks: all of them for SiLU inputs under decays of any size, with whole and partial
    last chunks; not all for tokens of 2^-12 to 2^12 that decays part, and none for decays that grow."""
    from llmss_b200.ops import _lib, cuda_impl as cu

    torch.manual_seed(8)
    lens, heads, qk_heads, d = [640, 33, 417, 512, 100, 290], 8, 4, 128
    T, B = sum(lens), len(lens)
    q, k, v = (torch.nn.functional.silu(torch.randn(T, n * d, device="cuda")) for n in (qk_heads, qk_heads, heads))
    if "unequal" in decay:
        v *= torch.exp2(torch.rand(T, 1, device="cuda") * 24 - 12)
    u, b = torch.rand(T, heads, device="cuda"), torch.randn(T, heads, device="cuda")
    g = {"mild": -0.3 * u, "slow": -0.01 * u, "strong": -3.0 - 9.0 * u, "resets": torch.where(u < 0.02, -20.0, -0.1 * u), "growing": 0.3 + 0.0 * u}[decay.split(",")[0]]
    batch, state, out = _batch(lens, [0] * B, range(B)), torch.empty(B, heads, d, d, device="cuda"), torch.empty(T, heads * d, device="cuda")
    lib, p = _lib.load(), cu._ptr
    scratch = torch.empty(lib.llmss_delta_scan_chunked_bytes(T, B, heads), dtype=torch.uint8, device="cuda")
    _lib.check(lib.llmss_delta_scan_chunked(p(q), q.stride(0), p(k), k.stride(0), p(v), v.stride(0), p(g), heads, p(b), heads, p(out), p(state), p(batch.cu_q),
                                            p(batch.seq_lens), p(batch.state_slots), B, max(lens), heads, qk_heads, d, d, 1e-6, d ** -0.5, 1, p(scratch), cu._stream()),
               "chunked")
    records = scratch.view(-1, heads, 13312)[:, :, 13312 - 4 * 29:13312 - 4 * 28].contiguous().view(torch.int32)[:, :, 0].cpu()
    firsts = [sum(lens[:i]) // 32 + i for i in range(B)]
    done = records[firsts]
    if stays:
        assert torch.equal(done, torch.tensor(lens, dtype=torch.int32)[:, None].expand(-1, heads))
    else:
        assert (done < torch.tensor(lens)[:, None]).any() and (decay != "growing" or not done.any())


@pytest.mark.parametrize("where", ["value", "key", "strength", "decay", "state", "huge value"])
def test_delta_over_chunks_bad_numbers(where, monkeypatch):
    """A value that is no number, or too large to scale, reaches what it reaches token by token: later tokens of its column (value, state) or of
    its head (key, strength, decay), never an earlier token or another head."""
    from llmss_b200.ops import cuda_impl as cu

    monkeypatch.setattr(cu, "_delta_over_chunks", lambda *a: True)
    torch.manual_seed(5)
    lens, heads, d = [100], 2, 128
    (q, k, v), b, S0 = _delta_inputs(lens, heads, 2, d, d, True)
    g, at, state = -0.3 * torch.rand(100, heads, device="cuda"), 45, S0.transpose(2, 3).contiguous().view(1, heads, d, d)
    clean_state = state.clone()
    call = lambda s: ops.delta_scan(q, k, v, g, b, _batch(lens, [3], [0]), s, heads, 2, d, d, unit_eps=1e-6, q_scale=0.25, beta_sigmoid=True).view(100, heads, d)
    clean = call(clean_state)
    bad = float("nan")
    if where == "value":
        v[at, d + 7] = bad
    elif where == "huge value":
        v[at, d + 7] = 1e35
    elif where == "key":
        k[at, d + 7] = bad
    elif where == "strength":
        b[at, 1] = bad
    elif where == "decay":
        g[at, 1] = bad
    else:
        state.view(1, heads, d, d)[0, 1, 7, 3] = bad
    got = call(state)
    assert torch.equal(got[:, 0], clean[:, 0]) and torch.equal(state[:, 0], clean_state[:, 0])
    from_ = 0 if where == "state" else at
    if where != "state":        # (the chunk of the bad number is computed token by token: other sums, the same bound)
        assert torch.equal(got[:32, 1], clean[:32, 1])
        assert _rel(got[32:at, 1], clean[32:at, 1].double().cpu()) < 1e-6
    if where in ("value", "state"):
        assert got[from_ + 1:, 1, 7].isnan().all()
        others = [i for i in range(d) if i != 7]
        assert _rel(got[:, 1, others], clean[:, 1, others].double().cpu()) < 1e-6
    elif where == "huge value":
        (S64,) = (S0.double().cpu(),)
        want, _ = _delta64(q, k, v, g, b, S64, lens, [3], heads, 2, d, d, True)
        assert _rel(got, want) < 1e-6
    else:
        assert got[at + 1:, 1].isnan().all()


@pytest.mark.parametrize("T,W,E,top,F,gated,skew", [(300, 128, 16, 4, 64, False, False), (1500, 256, 8, 2, 136, True, False), (513, 72, 5, 1, 40, False, True),
                                                    (1024, 64, 256, 8, 32, True, False), (700, 64, 3, 3, 264, False, False), (1, 64, 8, 2, 64, False, False)])
def test_experts_sorted_on_the_device(T, W, E, top, F, gated, skew):
    """Groups of no rows, of less and of more than a token tile, features off the 256-feature pairs, hidden sizes off the 64-column
    k-blocks, down matrices as a view of wider rows, a sum onto another result.  Every (token, expert) pair alone, with weight 1, row by row,
    so that a pair lost or misplaced at a group's edge is an error of the whole row; then all of them as weighted.  Bound: hidden
    rows rounded to bf16, 1e-2."""
    from llmss_b200.ops import cuda_impl as cu

    torch.manual_seed(T + E)
    dt = torch.bfloat16
    rows = 2 * F if gated else F
    h = torch.randn(T, W, device="cuda").to(dt)
    up = (torch.randn(E, rows, W, device="cuda") * W ** -0.5).to(dt)
    down = (torch.randn(W, 16 + E * F, device="cuda") * F ** -0.5).to(dt)[:, 16:]
    z = torch.randn(T, E, device="cuda") + (8.0 * (torch.arange(E, device="cuda") == 2) if skew else 0.0)
    ids, wts = ops.moe_route(z, E, top, 1, 1, 1.0)
    base = torch.randn(T, W, device="cuda")
    assert cu.moe_groups_on_device(h, up, down, gated)
    pairs = torch.empty(T, top, W, device="cuda", dtype=F64)
    for e in range(E):
        t, j = torch.nonzero(ids == e, as_tuple=True)
        x = h[t].double() @ up[e].double().t()
        x = torch.nn.functional.silu(x[:, 0::2]) * x[:, 1::2] if gated else torch.nn.functional.silu(x)
        pairs[t, j] = x @ down[:, e * F:(e + 1) * F].double().t()
    for j in range(top):
        one = torch.zeros_like(wts)
        one[:, j] = 1.0
        got = cu.moe_experts_grouped(h, ids, one, up, down, ops.ACT_SILU, gated)
        assert float(((got.double() - pairs[:, j]).norm(dim=1) / pairs[:, j].norm(dim=1)).max()) < 1e-2
    got = cu.moe_experts_grouped(h, ids, wts, up, down, ops.ACT_SILU, gated, base=base.clone())
    want = (wts.double()[:, :, None] * pairs).sum(1)
    assert _rel(got.double() - base.double(), want.cpu()) < 1e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,E,K,top,groups,keep,score,extra", [(1, 8, 8, 2, 1, 1, "softmax", False), (15, 16, 264, 4, 4, 2, "softmax", True), (17, 6, 40, 3, 3, 2, "sigmoid", True),
                                                               (33, 32, 2048, 4, 8, 4, "sigmoid", True), (100, 20, 520, 5, 1, 1, "softmax", False), (16, 32, 4096, 8, 8, 3, "softmax", True)])
def test_router_in_one_launch(T, E, K, top, groups, keep, score, extra, dtype):
    """Logits and routing together against the oracle's routing of 64-bit logits: tokens and experts short of a tile, widths short of a step.  Weights: 32-bit
    sums of K products of 16-bit numbers, 1e-5; a choice may differ only where two scores lie closer than that, and every other one is compared."""
    from llmss_b200.ops import cuda_impl as cu, reference as R

    torch.manual_seed(T + E)
    wide = torch.randn(T, K + 8, device="cuda").to(dtype)
    h = wide[:, 8:]
    w = (2 * torch.randn(E, K, device="cuda") * K ** -0.5).to(dtype)
    bias = torch.randn(E, device="cuda").to(dtype) if extra else None
    corr = 0.1 * torch.randn(E, device="cuda") if score == "sigmoid" else None
    z = h.double() @ w.double().t() + (bias.double() if extra else 0.0)
    kw = dict(score=score, correction=corr, group_top=min(2, E // groups) if score == "sigmoid" else 1)
    assert cu.moe_router_fused(h, w, bias, E)
    ids, wts, dense = cu.moe_router(h, w, bias, E, top, groups, keep, 1.5, dense=True, **kw)
    want_ids, want = R.moe_route(z.float().cpu(), E, top, groups, keep, 1.5, score, None if corr is None else corr.cpu(), kw["group_top"])
    got_ids, got = ids.cpu(), wts.cpu()
    full = torch.zeros(T, E).scatter_(1, got_ids.long(), got)
    assert torch.equal(full, dense.cpu())
    # choices that a difference of 1e-5 cannot turn: neighbours among the best `top` + 1 experts of the kept groups, and the last group kept and the first dropped
    zc = z.cpu()
    c = (torch.softmax(zc, -1) if score == "softmax" else torch.sigmoid(zc)) + (0.0 if corr is None else corr.cpu().double())
    gs = c.view(T, groups, -1).topk(kw["group_top"], -1).values.sum(-1).sort(-1, descending=True)
    kept = torch.zeros(T, groups, dtype=torch.bool).scatter_(1, gs.indices[:, :keep], True).repeat_interleave(E // groups, 1)
    best = c.masked_fill(~kept, -9.0).sort(-1, descending=True).values[:, :top + 1]
    decided = (best[:, :-1] - best[:, 1:] > 1e-5).all(1)
    if keep < groups:
        decided &= gs.values[:, keep - 1] - gs.values[:, keep] > 1e-5 * kw["group_top"]
    assert decided.float().mean() >= 0.9
    assert torch.equal(got_ids[decided], want_ids[decided])
    assert ((got - want).abs()[decided] <= 1e-5 * want.abs()[decided] + 1e-6).all()


@pytest.mark.parametrize("tile_rows", [32, 96, 224])
@pytest.mark.parametrize("T,top,E,W,F,gated", [(5, 2, 8, 256, 192, False), (95, 3, 6, 136, 72, True), (700, 4, 16, 512, 256, False)])
def test_grouped_tile_rows(T, top, E, W, F, gated, tile_rows):
    """Grouped products in narrow tiles: the same bits as in tiles of 256 rows (every number is the same sum over K)."""
    from llmss_b200.ops import cuda_impl as cu

    torch.manual_seed(T)
    dt = torch.bfloat16
    h = torch.randn(T, W, device="cuda").to(dt)
    up = (torch.randn(E, 2 * F if gated else F, W, device="cuda") * W ** -0.5).to(dt)
    down = (torch.randn(W, E * F, device="cuda") * F ** -0.5).to(dt)
    ids, wts = ops.moe_route(torch.randn(T, E, device="cuda"), E, top, 1, 1, 1.0)
    got, want = (cu.moe_experts_grouped(h, ids, wts, up, down, ops.ACT_SILU, gated, tile_rows=r) for r in (tile_rows, 256))
    assert torch.equal(got, want)


@pytest.mark.parametrize("T,top,E,skew", [(1, 2, 8, False), (300, 4, 16, False), (513, 1, 5, True), (1024, 8, 256, False), (1025, 3, 3, False), (4096, 2, 200, True)])
def test_pairs_sorted_by_expert(T, top, E, skew):
    """Places, row ranges and tile counts against a stable sort: single blocks and several, experts without pairs, a partial last block."""
    from llmss_b200.ops import _lib
    from llmss_b200.ops import cuda_impl as cu

    torch.manual_seed(T)
    P = T * top
    ids = torch.randint(0, E, (T, top), device="cuda", dtype=torch.int32)
    if skew:
        ids[torch.rand(T, top, device="cuda") < 0.9] = E // 2
    hist, table, inv = (torch.full((n,), -1, dtype=torch.int32, device="cuda") for n in (-(-P // 1024) * E, 2 * (E + 1), P))
    _lib.check(_lib.load().llmss_moe_group(cu._ptr(ids), P, E, cu._ptr(hist), cu._ptr(table), cu._ptr(inv), cu._stream()), "llmss_moe_group")
    counts = torch.bincount(ids.flatten().cpu(), minlength=E)
    order = torch.sort(ids.flatten().cpu(), stable=True).indices
    want = torch.empty(P, dtype=torch.long)
    want[order] = torch.arange(P)
    assert torch.equal(inv.cpu().long(), want)
    zero = torch.zeros(1, dtype=torch.long)
    assert torch.equal(table[:E + 1].cpu().long(), torch.cat([zero, counts.cumsum(0)]))
    assert torch.equal(table[E + 1:].cpu().long(), torch.cat([zero, ((counts + 255) // 256).cumsum(0)]))


def _scan64(q, k, v, a, bonus, before, lens, S0):
    """The recurrence of ops.reference.linear_scan in 64 bits; a [T, H, dk] decay factors; S0 per sequence [H, dk, dv]."""
    out, ends, at = torch.zeros_like(v), [], 0
    for n, S in zip(lens, S0):
        S = S.clone()
        for t in range(at, at + n):
            kv = k[t][:, :, None] * v[t][:, None, :]
            new = a[t][:, :, None] * S + kv
            read = (S + (bonus[:, :, None] * kv if bonus is not None else 0)) if before else new
            out[t] = torch.einsum("hkv,hk->hv", read, q[t])
            S = new
        ends.append(S)
        at += n
    return out, ends


@pytest.mark.parametrize("kind,dk,dv,heads,qk_heads,before,deep", [
    (2, 64, 64, 2, 2, True, 0), (2, 128, 128, 2, 2, False, 0), (1, 128, 64, 4, 2, False, 0), (0, 128, 128, 2, 2, False, 0), (2, 4, 1, 3, 3, False, 0),
    (2, 60, 70, 2, 2, True, 0), (1, 100, 130, 2, 1, True, 0), (0, 68, 3, 2, 2, False, 0), (2, 64, 64, 2, 2, True, 1), (2, 128, 72, 1, 1, False, 1),
    (1, 64, 16, 2, 2, False, 2)])
def test_linear_scan_over_chunks(kind, dk, dv, heads, qk_heads, before, deep):
    """Portions that end inside, at and behind a chunk, with and without a state, in packed order and with an inert sequence; strides
    off the 16-byte lines; ``deep``: decays past 2^-80 within half a sub-block (1), growth (2) -- the token-by-token form of a chunk.
    Bound: 32-bit sums, 2e-6 of the norm."""
    torch.manual_seed(dk * 7 + dv)
    lens, ctxs, slots = [64, 1, 130, 65, 200, 3], [0, 5, 7, 0, 64, 9], [4, 0, 2, 5, 1, -1]
    T = sum(lens)
    wide = lambda n: torch.randn(T, n + 3, device="cuda")[:, 1:n + 1]
    q, k, v = wide(qk_heads * dk), wide(qk_heads * dk), wide(heads * dv)
    bonus = torch.randn(heads, dk, device="cuda") * 0.5 if before else None
    scale = None
    if kind == 0:
        dec = torch.rand(heads, device="cuda") * 0.5 + 0.5
        a = dec.double().cpu().view(1, heads, 1).expand(T, heads, dk)
    else:
        n = heads if kind == 1 else heads * dk
        dec = -torch.exp(wide(n) - 1.0)
        if deep == 1:
            dec = torch.where(torch.rand(T, n, device="cuda") < 0.02, -300.0, dec)
        if deep == 2:
            dec = torch.where(torch.rand(T, n, device="cuda") < 0.01, 8.0, dec * 2)
        a = torch.exp(dec.double().cpu()).view(T, heads, -1).expand(T, heads, dk)
        scale = torch.rand(T, heads, device="cuda") + 0.5 if kind == 1 else None
    state = torch.randn(6, heads, dk, dv, device="cuda")
    S0 = [state[s].reshape(heads, dv, dk).transpose(1, 2).double().cpu() if c else torch.zeros(heads, dk, dv, dtype=F64) for s, c in zip(slots, ctxs)]
    rep = heads // qk_heads
    d = lambda x, n, w: x.double().cpu().reshape(T, n, w)
    vv = d(v, heads, dv) * (scale.double().cpu()[:, :, None] if scale is not None else 1.0)
    want, ends = _scan64(d(q, qk_heads, dk).repeat_interleave(rep, 1), d(k, qk_heads, dk).repeat_interleave(rep, 1), vv, a,
                         bonus.double().cpu() if before else None, before, lens, S0)
    before_state = state.clone()
    got = ops.linear_scan(q, k, v, dec, kind, _batch(lens, ctxs, slots), state, heads, qk_heads, dk, dv, bonus=bonus, v_scale=scale,
                          read_before=before)
    live = T - lens[-1]
    assert _rel(got[:live], want.reshape(T, -1)[:live]) < 2e-6
    for s, S in zip(slots[:-1], ends):
        assert _rel(state[s].reshape(heads, dv, dk).transpose(1, 2), S) < 2e-6
    assert torch.equal(state[3], before_state[3])        # a slot that no sequence names


def _scan_case(seed, kind, dk, dv, heads, lens, before, decay):
    """Inputs of a recurrence over fresh sequences and its float64 results; decay(shape) gives the log decays."""
    torch.manual_seed(seed)
    T = sum(lens)
    q, k, v = (torch.randn(T, heads * n, device="cuda") for n in (dk, dk, dv))
    logs = decay((heads,) if kind == 0 else (T, heads) if kind == 1 else (T, heads * dk))
    dec = torch.exp(logs) if kind == 0 else logs
    factors = dec.double().cpu() if kind == 0 else torch.exp(dec.double().cpu())
    a = factors.view(1, heads, 1).expand(T, heads, dk) if kind == 0 else factors.view(T, heads, -1).expand(T, heads, dk)
    bonus = torch.randn(heads, dk, device="cuda") * 0.5 if before else None

    def want():
        d = lambda x, w: x.double().cpu().reshape(T, heads, w)
        return _scan64(d(q, dk), d(k, dk), d(v, dv), a, bonus.double().cpu() if before else None, before, lens,
                       [torch.zeros(heads, dk, dv, dtype=F64)] * len(lens))

    def run():
        state = torch.zeros(len(lens), heads, dk, dv, device="cuda")
        out = ops.linear_scan(q, k, v, dec, kind, _batch(lens, [0] * len(lens), list(range(len(lens)))), state, heads, heads, dk, dv, bonus=bonus,
                              read_before=before)
        return out, state.reshape(len(lens), heads, dv, dk).transpose(2, 3)

    return (q, k, v, dec, bonus), want, run


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("before", [False, True])
@pytest.mark.parametrize("dk", [64, 128])
@pytest.mark.parametrize("log", [-4.0, -5.0, -6.0, -6.8, -7.0, -8.0, -8.6, -9.0, "one", "near"])
def test_linear_scan_strong_decays(kind, before, dk, log):
    """Decays that leave little of a state after a few tokens, all of them or one channel in 64 (one head in two): on both sides of what
    the products take, and around it.  The rows at sub-block starts are looked at one by one: what they see of the sub-block before
    them has full weight.  Bound: 32-bit sums, 2e-6 of the norm."""
    def decay(shape):
        if log == "one":
            x = torch.full(shape, -0.4, device="cuda")
            x[..., 1::64 if kind == 2 else 2] = -7.0
            return x
        if log == "near":
            return -torch.exp(torch.randn(shape, device="cuda") * 0.2 + 1.9)
        return torch.full(shape, log, device="cuda")

    lens = [200, 130]
    _, want, run = _scan_case(dk + kind, kind, dk, 40, 2, lens, before, decay)
    (w, ends), (got, state) = want(), run()
    w = w.reshape(got.shape)
    assert _rel(got, w) < 2e-6
    rows = [at + t for at, n in zip((0, 200), lens) for t in range(16 if before else 0, n, 16)]
    err = (got.double().cpu() - w)[rows].norm(dim=1) / w[rows].norm(dim=1)
    assert float(err.max()) < 2e-6
    assert _rel(state, torch.stack(ends)) < 2e-6


@pytest.mark.parametrize("kind,dk,before", [(2, 64, True), (2, 128, False), (1, 128, False), (0, 64, False)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_linear_scan_keeps_a_bad_value_behind_its_token(kind, dk, before, bad):
    """A value that is no number, or infinite, in the middle of a sub-block: earlier tokens and other columns are as without it."""
    (q, k, v, dec, bonus), want, run = _scan_case(3, kind, dk, 40, 2, [200], before, lambda s: -torch.rand(s, device="cuda") * 0.5)
    w = want()[0]
    v[77, 5] = bad
    got = run()[0].reshape(200, 2, 40)
    assert _rel(got[:77], w[:77]) < 2e-6
    assert not torch.isfinite(got[78:, 0, 5]).any()
    got[:, 0, 5], w[:, 0, 5] = 0.0, 0.0
    assert _rel(got, w) < 2e-6


@pytest.mark.parametrize("kind,dk,before", [(2, 64, True), (2, 128, False), (1, 128, False), (0, 20, False)])
@pytest.mark.parametrize("floor", [None, 0, 64])
def test_linear_scan_long_and_short_portions_together(kind, dk, before, floor, monkeypatch):
    """A batch of whole chunks, of lengths around a chunk and of single tokens, every way that the rule can send it: all token by token,
    all over chunks, and split at 64 tokens.  Fresh sequences; every state is written once.  Bound: 32-bit sums, 2e-6 of the norm."""
    from llmss_b200.ops import cuda_impl as cu

    monkeypatch.setattr(cu, "_scan_floor", lambda *a: floor)
    lens = [1, 130, 1, 63, 64, 65, 2, 1, 200, 16, 1]
    _, want, run = _scan_case(dk, kind, dk, 24, 2, lens, before, lambda s: -torch.exp(torch.randn(s, device="cuda") - 1.0))
    (w, ends), (got, state) = want(), run()
    assert _rel(got, w.reshape(got.shape)) < 2e-6
    for i, S in enumerate(ends):
        assert _rel(state[i], S) < 2e-6, lens[i]


@pytest.mark.parametrize("kind,dk,before", [(2, 64, True), (2, 128, False), (1, 128, False), (0, 128, False)])
@pytest.mark.parametrize("log", ["mild", "slow", -0.05, -2.0, -6.5, -9.0, "one"])
def test_linear_scan_over_chunks_rounds_like_token_by_token(kind, dk, before, log, monkeypatch):
    """The error against 64 bits is not above the token-serial form's, outputs and states, for decays from a long memory to none (-9: chunks
    that run token by token).  Both are the norm of some 10^4 independent roundings, which repeats to about 2 % from seed to seed; bound 5 %."""
    from llmss_b200.ops import cuda_impl as cu

    def decay(shape):
        if log == "mild":
            return -torch.exp(torch.randn(shape, device="cuda") - 1.0)
        if log == "slow":
            return -torch.exp(torch.randn(shape, device="cuda") * 0.7 - 3.0)
        if log == "one":
            x = torch.full(shape, -0.4, device="cuda")
            x[..., 1::64 if kind == 2 else 2] = -7.0
            return x
        return torch.full(shape, log, device="cuda")

    _, want, run = _scan_case(1, kind, dk, 64, 4, [256, 130, 64], before, decay)
    w, ends = want()
    ends = torch.stack(ends)
    errors = []
    for floor in (0, None):
        monkeypatch.setattr(cu, "_scan_floor", lambda *a: floor)
        got, state = run()
        errors.append((_rel(got, w.reshape(got.shape)), _rel(state, ends)))
    assert errors[0][0] < 1.05 * errors[1][0] and errors[0][1] < 1.05 * errors[1][1], errors


@pytest.mark.parametrize("kind,dk,before", [(2, 64, True), (2, 128, False), (1, 128, False), (0, 64, False)])
def test_linear_scan_portions_agree_across_the_rule(kind, dk, before):
    """The same 192 tokens in portions of 96 and 96, 95 and 97, and whole: equal to rounding, 2e-6 of the norm."""
    (q, k, v, dec, bonus), want, _ = _scan_case(9, kind, dk, 24, 2, [192], before, lambda s: -torch.rand(s, device="cuda"))
    w = want()[0].reshape(192, -1)
    for cut in (96, 95, 192):
        state, outs = torch.zeros(1, 2, dk, 24, device="cuda"), []
        for lo, hi in ((0, cut), (cut, 192)):
            if hi > lo:
                part = [x[lo:hi] for x in (q, k, v)]
                outs.append(ops.linear_scan(*part, dec if kind == 0 else dec[lo:hi], kind, _batch([hi - lo], [lo], [0]), state, 2, 2, dk, 24,
                                            bonus=bonus, read_before=before))
        assert _rel(torch.cat(outs), w) < 2e-6, cut


@pytest.mark.parametrize("T,H,k,n,xs,form", [(129, 3, 128, 128, None, None), (300, 5, 64, 192, 72, "row"), (513, 2, 192, 128, 256, "elem"), (257, 16, 40, 24, None, "f32"),
                                             (2000, 33, 128, 136, None, "row"), (130, 2, 8, 40, None, "row"), (385, 3, 72, 8, 80, "f32")])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_per_head_products_at_prompt_sizes(T, H, k, n, xs, form, dt):
    """Tokens, features and contraction off the tile sizes, features that end inside a warp's 32 (the other lanes only take part in the
    loads from tensor memory), heads as column ranges of wider rows, results between other columns, the factor per token and head or per
    element.  Bound: one rounding to 16 bits of 32-bit sums (2^-8 / 2^-11 of a value), 1e-6 in 32-bit."""
    torch.manual_seed(T)
    xs = xs or k
    x = torch.randn(T, H * xs, device="cuda").to(dt)
    w = (torch.randn(H, n, k, device="cuda") * k ** -0.5).to(dt)
    row = torch.rand(T, H + 1, device="cuda")[:, 1:] if form == "row" else None
    elem = torch.rand(T, H * n, device="cuda") if form == "elem" else None
    out = torch.zeros(T, H * (n + 8), device="cuda", dtype=F32 if form == "f32" else dt)
    ops.heads_matmul(x, w, H, k, n, False, row_scale=row, x_head_stride=xs, elem_scale=elem, out=out, out_head_stride=n + 8)
    want = torch.einsum("thk,hnk->thn", x.view(T, H, xs)[:, :, :k].double(), w.double())
    if row is not None:
        want = want * row.double()[:, :, None]
    if elem is not None:
        want = want * elem.double().view(T, H, n)
    got = out.view(T, H, n + 8)
    assert _rel(got[:, :, :n], want.cpu()) < (1e-6 if form == "f32" else 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11)
    assert not got[:, :, n:].any()


@pytest.mark.parametrize("C,groups,act,first,skip", [(256, 4, 1, False, False), (128, 1, 2, False, True), (512, 2, 1, True, True), (1024, 1, 0, False, False),
                                                     (3072, 3, 1, True, False), (96, 1, 1, False, False), (512, 1, None, False, False)])
@pytest.mark.parametrize("T", [1, 37])
@pytest.mark.parametrize("off", [0, 1])
def test_gated_norm_groups(C, groups, act, first, skip, T, off):
    """Groups that a warp (or half of one) holds in registers, odd group sizes, columns off the 16-byte lines (``off``).
    Bound: 32-bit arithmetic, 2e-6 of the norm."""
    torch.manual_seed(C + T)
    wide = lambda: torch.randn(T, C + 8, device="cuda")[:, off:off + C]
    o, gate, w, x = wide(), wide(), torch.rand(C, device="cuda") + 0.5, wide()
    d = torch.randn(4, device="cuda")
    got = ops.gated_rmsnorm(o, gate if act is not None else None, act or 0, w, groups, 1e-6, first, skip_x=x if skip else None,
                            skip_d=d if skip else None)
    y = o.double()
    if skip:
        y = y + (x.double().reshape(T, 4, C // 4) * d.double()[None, :, None]).reshape(T, C)
    g = 1.0
    if act is not None:
        g = {0: lambda z: z, 1: torch.nn.functional.silu, 2: torch.sigmoid}[act](gate.double())
    if first:
        y = y * g
    y = y.reshape(T, groups, -1)
    y = (y * torch.rsqrt(y.square().mean(-1, keepdim=True) + 1e-6)).reshape(T, C) * w.double()
    assert _rel(got, (y if first else y * g).cpu()) < 2e-6


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("act", [ops.ACT_NONE, ops.ACT_SILU, ops.ACT_GELU_ERF])
def test_convolution_rows(taps, act):
    """Portions around the blocks of 8 and the chunks of 16 rows, shorter than the taps, with and without a tail, an inert row.
    Bound: 32-bit arithmetic, 2e-6 of the norm; tails are copies."""
    torch.manual_seed(taps)
    lens, ctxs, slots, C = [1, 8, 15, 17, 40, 2, 5], [3, 0, 5, 0, 9, 1, 4], [0, 3, 1, 2, 6, 4, -1], 132
    T = sum(lens)
    u, w, b = torch.randn(T, C + 4, device="cuda")[:, :C], torch.randn(C, taps, device="cuda"), torch.randn(C, device="cuda")
    state = torch.randn(7, max(1, taps - 1), C, device="cuda") if taps > 1 else None
    old = state.clone() if taps > 1 else None
    got = ops.causal_conv(u, w, b, act, _batch(lens, ctxs, slots), state)
    at = 0
    for n, c, s in zip(lens, ctxs, slots):
        if s >= 0:
            hist = (old[s] if c else torch.zeros_like(old[s])) if taps > 1 else u[:0]
            full = torch.cat([hist, u[at:at + n]]).double()
            y = sum(full[j:j + n] * w[:, j].double() for j in range(taps)) + b.double()
            y = {ops.ACT_NONE: lambda z: z, ops.ACT_SILU: torch.nn.functional.silu, ops.ACT_GELU_ERF: torch.nn.functional.gelu}[act](y)
            assert _rel(got[at:at + n], y.cpu()) < 2e-6, (n, c)
            if taps > 1:
                assert torch.equal(state[s], full[-(taps - 1):].float())
        at += n


@pytest.mark.parametrize("H", [256, 1600, 2048, 2056, 4096, 5120, 8192])
@pytest.mark.parametrize("kind", [ops.NORM_LAYER, ops.NORM_RMS])
@pytest.mark.parametrize("extra", [0, 1, 2])
def test_norm_rows_at_prompt_sizes(H, kind, extra):
    """Rows off the warp's and the block's multiples, with a residual and a second addend.  The same rounding points as the oracle:
    bound of one bf16 rounding of the result, 2^-8 of a value, and of the stored sum exactly."""
    from llmss_b200.ops import reference as R

    torch.manual_seed(H)
    M, dt = 601, torch.bfloat16
    x, r, x2 = (torch.randn(M, H, device="cuda").to(dt) for _ in range(3))
    w, b = (torch.randn(H, device="cuda").to(dt) for _ in range(2))
    got, res = ops.norm_residual(x, r if extra else None, w, b if kind == ops.NORM_LAYER else None, 1e-5, kind, x2=x2 if extra == 2 else None)
    total = x.float() + (x2.float() if extra == 2 else 0) + (r.float() if extra else 0)
    total = total.to(dt)
    assert torch.equal(res, total)
    want, _ = R.norm_residual(total.double().cpu(), None, w.cpu(), b.cpu() if kind == ops.NORM_LAYER else None, 1e-5, kind, out_dtype=F32)
    assert _rel(got, want.double()) < 2.0 ** -8


@pytest.mark.parametrize("H", [8, 256, 1600, 2048, 2056, 4096, 4104, 5120, 8192])
@pytest.mark.parametrize("kind", [ops.NORM_LAYER, ops.NORM_RMS])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_a_norm_row_is_the_same_in_any_batch(H, kind, dt):
    """Prompt sizes and a block per row sum in the same order: equal bits."""
    torch.manual_seed(H)
    M = 603
    x, r, x2 = (torch.randn(M, H, device="cuda").to(dt) for _ in range(3))
    w, b = (torch.randn(H, device="cuda").to(dt) for _ in range(2))
    b = b if kind == ops.NORM_LAYER else None
    whole = ops.norm_residual(x, r, w, b, 1e-5, kind, x2=x2)
    for lo in range(0, M, 201):
        rows = slice(lo, lo + 201)
        part = ops.norm_residual(x[rows], r[rows], w, b, 1e-5, kind, x2=x2[rows])
        for a, c in zip(whole, part):
            assert torch.equal(a[rows], c)


@pytest.mark.parametrize("kind,dk,dv,heads,qk_heads,before", [
    (2, 64, 64, 2, 2, True), (0, 128, 128, 16, 16, False), (1, 128, 64, 4, 2, False), (2, 4, 1, 3, 3, False), (2, 36, 70, 2, 2, True),
    (1, 100, 130, 2, 1, True), (0, 32, 33, 2, 2, False), (2, 128, 7, 64, 64, True)])
def test_linear_scan_one_token(kind, dk, dv, heads, qk_heads, before):
    """A token per sequence: columns off a warp's and a block's multiples, key sizes that leave lanes idle, few and many blocks, fresh
    and running states (a fresh one holds NaN before), an inert sequence, strides off the 16-byte lines.  Bound: 32-bit sums, 2e-6."""
    torch.manual_seed(dk * 7 + dv)
    ctxs, slots = [5, 0, 9, 64, 3, 1], [4, 0, 2, 5, 1, -1]
    lens = [1] * len(ctxs)
    T = len(lens)
    wide = lambda n: torch.randn(T, n + 3, device="cuda")[:, 1:n + 1]
    q, k, v = wide(qk_heads * dk), wide(qk_heads * dk), wide(heads * dv)
    bonus = torch.randn(heads, dk, device="cuda") * 0.5 if before else None
    scale = torch.rand(T, heads, device="cuda") + 0.5 if kind == 1 else None
    if kind == 0:
        dec = torch.rand(heads, device="cuda") * 0.5 + 0.5
        a = dec.double().cpu().view(1, heads, 1).expand(T, heads, dk)
    else:
        dec = -torch.exp(wide(heads if kind == 1 else heads * dk) - 1.0)
        a = torch.exp(dec.double().cpu()).view(T, heads, -1).expand(T, heads, dk)
    state = torch.randn(6, heads, dk, dv, device="cuda")
    state[0] = float("nan")
    S0 = [state[s].reshape(heads, dv, dk).transpose(1, 2).double().cpu() if c and s >= 0 else torch.zeros(heads, dk, dv, dtype=F64)
          for s, c in zip(slots, ctxs)]
    rep = heads // qk_heads
    d = lambda x, n, w: x.double().cpu().reshape(T, n, w)
    vv = d(v, heads, dv) * (scale.double().cpu()[:, :, None] if scale is not None else 1.0)
    want, ends = _scan64(d(q, qk_heads, dk).repeat_interleave(rep, 1), d(k, qk_heads, dk).repeat_interleave(rep, 1), vv, a,
                         bonus.double().cpu() if before else None, before, lens, S0)
    untouched = state[3].clone()
    got = ops.linear_scan(q, k, v, dec, kind, _batch(lens, ctxs, slots), state, heads, qk_heads, dk, dv, bonus=bonus, v_scale=scale,
                          read_before=before)
    assert _rel(got[:T - 1], want.reshape(T, -1)[:T - 1]) < 2e-6
    for s, S in zip(slots[:-1], ends):
        assert _rel(state[s].reshape(heads, dv, dk).transpose(1, 2), S) < 2e-6
    assert torch.equal(state[3], untouched)        # a slot that no sequence names
