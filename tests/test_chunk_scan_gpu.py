"""The chunked form of the two recurrences with a decay per key channel, against float64 and against the token-by-token scans."""
import numpy as np
import pytest
import torch

import kernel_refs

pytestmark = pytest.mark.gpu
DEV = "cuda"


def g64(*shape, seed=0, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed), dtype=torch.float64) * scale


def i32(v):
    return torch.tensor([int(x) for x in v], dtype=torch.int32, device=DEV)


# A sum of up to 64 state channels plus 32 tokens, each term rounded once or twice: some hundred roundings of terms no larger than the
# results' scale (values of about 10 here).
TOL = 2e-5


@pytest.mark.parametrize("lens", [[2], [64], [1, 96, 31, 32, 33, 2], [257, 100]])
@pytest.mark.parametrize("H,dim,vdim", [(2, 64, 128), (2, 40, 24), (2, 1, 4), (2, 24, 68)])
@pytest.mark.parametrize("form", ["logits", "steep", "constant"])
def test_gated_linear_attention(lens, H, dim, vdim, form, monkeypatch):
    from dotllm_b200.kernels import ops
    monkeypatch.setattr(ops, "CHUNK_MIN_TOKENS", 2)
    T, tau = sum(lens), 5.0
    proj = g64(T, 2 * H * dim + H * vdim + 4, seed=1).to(torch.bfloat16).to(DEV)
    q, k, v = proj[:, :H * dim], proj[:, H * dim:2 * H * dim], proj[:, 2 * H * dim:2 * H * dim + H * vdim]
    z = None if form == "constant" else (g64(T, H * dim, seed=3) * (80.0 if form == "steep" else 2.0)).float().to(DEV)
    bias = (torch.linspace(0.3, 1.0, H) if z is None else g64(H * dim, seed=5)).float().to(DEV)
    slots = [4, 0, 3, 1, 5, 2][:len(lens)]
    state0 = g64(7, H, dim, vdim, seed=6).float().to(DEV)
    cu = i32([0] + list(np.cumsum(lens)))

    def run(most):
        s = state0.clone()
        return ops.gla_scan(q, k, v, z, bias, cu, i32(slots), s, H, dim, vdim, 0.3, tau, max_new=most), s

    got, state = run(max(lens))
    scan, _ = run(1)
    act = (lambda t: t * torch.sigmoid(t)) if z is None else (lambda t: t)
    at = 0
    for n, slot in zip(lens, slots):
        rows = slice(at, at + n)
        qd, kd = act(q[rows].double()).view(n, H, dim) * 0.3, act(k[rows].double()).view(n, H, dim)
        vd, s = act(v[rows].double()).view(n, H, vdim), state0[slot].double()
        alpha = bias.double().view(1, H, 1).expand(n, H, dim) if z is None else \
            (torch.nn.functional.logsigmoid((z[rows] + bias).double()) / tau).exp().view(n, H, dim)
        want = torch.empty(n, H, vdim, dtype=torch.float64, device=DEV)
        for t in range(n):
            s = alpha[t].unsqueeze(-1) * s + kd[t].unsqueeze(-1) * vd[t].unsqueeze(1)
            want[t] = (s * qd[t].unsqueeze(-1)).sum(1)
        scale = 1.0 + float(want.abs().max())
        assert float((got[rows].view(n, H, vdim) - want).abs().max()) < TOL * scale
        assert float((state[slot] - s).abs().max()) < TOL * (1 + float(s.abs().max()))
        # no further off than the scan, beyond the last bits
        far = lambda x: float((x[rows].view(n, H, vdim) - want).norm() / want.norm())
        assert far(got) < 1.5 * far(scan) + 1e-7
        at += n
    others = [i for i in range(7) if i not in slots]
    assert torch.equal(state[others], state0[others])


@pytest.mark.parametrize("H,G,dim,vdim", [(4, 2, 64, 128), (2, 2, 24, 20), (1, 1, 8, 4), (6, 2, 40, 68), (40, 40, 64, 128)])
@pytest.mark.parametrize("head_decay", [False, True])
def test_delta_rule(H, G, dim, vdim, head_decay, monkeypatch):
    """(Forty heads of 128 value channels: the walk over 32 columns a block; the others: over 16.)"""
    from dotllm_b200.kernels import ops
    monkeypatch.setattr(ops, "CHUNK_MIN_TOKENS", 2)
    K, lens = 4, [70, 1, 97, 32, 5]
    C, T, n_state = 2 * G * dim + H * vdim, sum(lens), H * dim * vdim
    taps = g64(C, K, seed=1, scale=0.5).to(torch.bfloat16)
    decays = H if head_decay else H * dim
    dt_bias, a_log = g64(decays, seed=2).float(), g64(H, seed=3, scale=0.5).float()
    x = g64(T, C + H, seed=10).to(torch.bfloat16)
    z = g64(T, decays, seed=20).float()
    memory = g64(6, n_state + (K - 1) * C, seed=4).float()
    slots = [4, 1, 5, 0, 2]
    seq, cu = [i for i, n in enumerate(lens) for _ in range(n)], [0] + list(np.cumsum(lens))
    gx = x.to(DEV)

    def run(most):
        m = memory.clone().to(DEV)
        return ops.delta_rule(gx, taps.to(DEV), gx[:, C:], z.to(DEV), dt_bias.to(DEV), a_log.to(DEV), i32(seq), i32(cu), i32(slots), m, H, G, dim, vdim,
                              dim ** -0.5, 1e-6, head_decay=head_decay, max_new=most), m

    got, mem = run(max(lens))
    scan, scan_mem = run(1)
    if H > 6:                                              # the oracle takes too long: the scan, which it has been held to at other sizes
        want, want_mem = scan.cpu(), scan_mem.cpu()
    else:
        want_mem = memory.clone()
        want = kernel_refs.delta_rule(x, taps, x[:, C:], z.repeat_interleave(dim, 1) if head_decay else z,
                                      dt_bias.repeat_interleave(dim) if head_decay else dt_bias, a_log, torch.tensor(seq), torch.tensor(cu),
                                      torch.tensor(slots), want_mem, H, G, dim, vdim, dim ** -0.5, 1e-6)
    scale = 1.0 + float(want.abs().max())
    assert float((got.cpu() - want).abs().max()) < 3 * TOL * scale
    assert float((mem.cpu() - want_mem).abs().max()) < 3 * TOL * (1 + float(want_mem.abs().max()))
    assert float((got - scan).abs().max()) < 3 * TOL * scale
    assert torch.equal(mem[3], memory[3].to(DEV)) and torch.equal(mem[:, n_state:], scan_mem[:, n_state:])


def no_worse(got, state, clean, scan, scan_state, before):
    """Rows of the tokens before keep their bits; what is no number is so exactly where the scan has it, the rest agrees with the scan."""
    assert torch.equal(got[before], clean[before])
    for a, b in ((got, scan), (state, scan_state)):
        fine = torch.isfinite(b)
        assert torch.equal(torch.isfinite(a), fine) and not bool(fine.all())
        assert float((a - b)[fine].abs().max()) < TOL * (1 + float(b[fine].abs().max()))


@pytest.mark.parametrize("what", ["v", "k", "q", "z"])
@pytest.mark.parametrize("token", [0, 45, 63, 64])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_linear_attention_of_a_token_that_is_no_number(what, token, value, monkeypatch):
    from dotllm_b200.kernels import ops
    monkeypatch.setattr(ops, "CHUNK_MIN_TOKENS", 2)
    H, dim, vdim, lens = 2, 40, 72, [100, 70]
    T = sum(lens)
    proj = g64(T, 2 * H * dim + H * vdim, seed=1).to(torch.bfloat16).to(DEV)
    z, bias = (g64(T, H * dim, seed=3) * 2).float().to(DEV), g64(H * dim, seed=5).float().to(DEV)
    state0 = g64(2, H, dim, vdim, seed=6).float().to(DEV)

    def run(most):
        s = state0.clone()
        q, k, v = proj[:, :H * dim], proj[:, H * dim:2 * H * dim], proj[:, 2 * H * dim:]
        return ops.gla_scan(q, k, v, z, bias, i32([0, 100, 170]), i32([1, 0]), s, H, dim, vdim, 0.3, 5.0, max_new=most), s

    clean, clean_state = run(100)
    if what == "z":
        z[token, 3] = float("nan")                         # (an infinite logit is a decay of 0 or 1)
    else:
        proj[token, {"q": 0, "k": H * dim, "v": 2 * H * dim}[what] + 5] = value
    got, state = run(100)
    scan, scan_state = run(1)
    if what == "q":                                        # only its own row
        assert torch.equal(state, clean_state) and torch.equal(torch.isfinite(got), torch.isfinite(scan))
        assert torch.equal(got[[t for t in range(T) if t != token]], clean[[t for t in range(T) if t != token]])
        return
    no_worse(got, state, clean, scan, scan_state, list(range(token)) + list(range(100, T)))


@pytest.mark.parametrize("what", ["v", "k", "b", "z"])
@pytest.mark.parametrize("token", [0, 45, 63, 64])
@pytest.mark.parametrize("H,G", [(4, 2), (40, 40)])
def test_delta_rule_of_a_token_that_is_no_number(what, token, H, G, monkeypatch):
    """(Forty heads: the walk over 32 columns a block.)"""
    from dotllm_b200.kernels import ops
    monkeypatch.setattr(ops, "CHUNK_MIN_TOKENS", 2)
    dim, vdim, K, lens = 64, 128, 4, [100, 70]
    C, T, n_state = 2 * G * dim + H * vdim, sum(lens), H * dim * vdim
    taps, dt_bias, a_log = g64(C, K, seed=1, scale=0.5).to(torch.bfloat16).to(DEV), g64(H * dim, seed=2).float().to(DEV), g64(H, seed=3, scale=0.5).float().to(DEV)
    x, z = g64(T, C + H, seed=10).to(torch.bfloat16).to(DEV), g64(T, H * dim, seed=20).float().to(DEV)
    memory = g64(2, n_state + (K - 1) * C, seed=4).float().to(DEV)
    seq = i32([0] * 100 + [1] * 70)

    def run(most):
        m = memory.clone()
        o = ops.delta_rule(x, taps, x[:, C:], z, dt_bias, a_log, seq, i32([0, 100, 170]), i32([1, 0]), m, H, G, dim, vdim, dim ** -0.5, 1e-6, max_new=most)
        return o, m[:, :n_state].contiguous()

    clean, _ = run(100)
    if what == "z":
        z[token, 3] = float("nan")
    else:
        x[token, {"v": 2 * G * dim, "k": G * dim, "b": C}[what] + 1] = float("inf") if what == "v" else float("nan")
    got, state = run(100)
    scan, scan_state = run(1)
    no_worse(got, state, clean, scan, scan_state, list(range(token)) + list(range(100, T)))


def gla_call(lens, H, dim, vdim, seed=1):
    from dotllm_b200.kernels import ops
    T = sum(lens)
    proj = g64(T, 2 * H * dim + H * vdim, seed=seed).to(torch.bfloat16).to(DEV)
    z, bias = (g64(T, H * dim, seed=3) * 2).float().to(DEV), g64(H * dim, seed=5).float().to(DEV)
    states = g64(len(lens), H, dim, vdim, seed=6).float().to(DEV)

    def run(at, most):
        """Sequences ``at`` of them, in this order."""
        rows = torch.cat([torch.arange(sum(lens[:b]), sum(lens[:b + 1])) for b in at]).to(DEV)
        p, s = proj[rows], states[at].clone()
        q, k, v = p[:, :H * dim], p[:, H * dim:2 * H * dim], p[:, 2 * H * dim:]
        cu, zz = i32([0] + list(np.cumsum([lens[b] for b in at]))), z[rows]
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        out = ops.gla_scan(q, k, v, zz, bias, cu, i32(range(len(at))), s, H, dim, vdim, 0.3, 5.0, max_new=most)
        return out, s, torch.cuda.max_memory_allocated() - before
    return run, H * (32 * 96 + 64 + 64 * vdim)


def delta_call(lens, H, dim, vdim, K=4):
    from dotllm_b200.kernels import ops
    C, T, n_state = (2 * dim + vdim) * H, sum(lens), H * dim * vdim
    taps, dt_bias, a_log = g64(C, K, seed=1, scale=0.5).to(torch.bfloat16).to(DEV), g64(H, seed=2).float().to(DEV), g64(H, seed=3, scale=0.5).float().to(DEV)
    x, z = torch.randn(T, C + H, generator=torch.Generator().manual_seed(9)).to(torch.bfloat16).to(DEV), g64(T, H, seed=20).float().to(DEV)
    memory = g64(len(lens), n_state + (K - 1) * C, seed=4).float().to(DEV)

    def run(at, most):
        rows = torch.cat([torch.arange(sum(lens[:b]), sum(lens[:b + 1])) for b in at]).to(DEV)
        p, zz, m = x[rows], z[rows], memory[at].clone()
        seq, cu = i32([i for i, b in enumerate(at) for _ in range(lens[b])]), i32([0] + list(np.cumsum([lens[b] for b in at])))
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        out = ops.delta_rule(p, taps, p[:, C:], zz, dt_bias, a_log, seq, cu, i32(range(len(at))), m, H, H, dim, vdim, dim ** -0.5, 1e-6,
                             head_decay=True, max_new=most)
        return out, m, torch.cuda.max_memory_allocated() - before
    return run, H * 96 * 96


@pytest.mark.parametrize("call", [gla_call, delta_call])
@pytest.mark.parametrize("pieces", [1, 3, 7])
def test_windows_of_chunks_give_the_same_bits(call, pieces, monkeypatch):
    from dotllm_b200.kernels import ops
    monkeypatch.setattr(ops, "CHUNK_MIN_TOKENS", 2)
    lens = [1, 96, 31, 130, 2, 64, 33]
    run, floats = call(lens, 3, 40, 72)
    out, state, _ = run(list(range(7)), 130)
    assert torch.equal(run(list(range(7)), 2)[0], out)         # the most tokens of a sequence choose the form, nothing else
    monkeypatch.setattr(ops, "CHUNK_SCRATCH_BYTES", 4 * floats * pieces + 3)
    got, got_state, _ = run(list(range(7)), 130)
    assert torch.equal(got, out) and torch.equal(got_state, state)
    monkeypatch.setattr(ops, "CHUNK_SCRATCH_BYTES", 4 * floats - 1)      # not one piece: token by token
    assert torch.equal(run(list(range(7)), 130)[0], run(list(range(7)), 1)[0])


@pytest.mark.parametrize("call", [gla_call, delta_call])
def test_scratch_follows_the_tokens(call):
    """A prompt beside many single tokens takes the room of its own chunks and a piece for each of the others, and gets the bits it has alone."""
    lens = [1] * 20 + [1500] + [1] * 27
    run, floats = call(lens, 32, 64, 128)
    out, state, peak = run(list(range(48)), 1500)
    alone, alone_state, _ = run([20], 1500)
    assert torch.equal(out[20:1520], alone) and torch.equal(state[20], alone_state[0])
    _, _, scan_peak = run(list(range(48)), 1)
    assert peak - scan_peak < 0.2 * 2 ** 30
    assert peak - scan_peak <= 4 * floats * ((sum(lens) + 31 * 48) // 32) + (4 << 20)


@pytest.mark.parametrize("K", [1, 2, 3, 4])
@pytest.mark.parametrize("dim", [16, 32, 64])
@pytest.mark.parametrize("head_decay", [False, True])
def test_preparation_of_prompts(K, dim, head_decay, monkeypatch):
    """Fewer taps than the kernel's four places, heads of 4, 8 and 16 lanes, tokens that do not fill a block, sequences shorter than the taps."""
    from dotllm_b200.kernels import ops
    monkeypatch.setattr(ops, "CHUNK_MIN_TOKENS", 2)
    H, G, vdim, lens = 4, 2, 36, [37, 1, 2, 50, 3]
    C, T, n_state = 2 * G * dim + H * vdim, sum(lens), H * dim * vdim
    decays = H if head_decay else H * dim
    taps = g64(C, K, seed=1, scale=0.5).to(torch.bfloat16)
    dt_bias, a_log = g64(decays, seed=2).float(), g64(H, seed=3, scale=0.5).float()
    x, z = g64(T, C + H, seed=10).to(torch.bfloat16), g64(T, decays, seed=20).float()
    memory = g64(6, n_state + (K - 1) * C, seed=4).float()
    slots, seq, cu = [4, 1, 5, 0, 2], [i for i, n in enumerate(lens) for _ in range(n)], [0] + list(np.cumsum(lens))
    gx, gm = x.to(DEV), memory.clone().to(DEV)
    assert gx.stride(0) % 4 == 0 and gm.stride(0) % 4 == 0     # the kernel's four channels a thread
    got = ops.delta_rule(gx, taps.to(DEV), gx[:, C:], z.to(DEV), dt_bias.to(DEV), a_log.to(DEV), i32(seq), i32(cu), i32(slots), gm, H, G, dim, vdim,
                         dim ** -0.5, 1e-6, head_decay=head_decay, max_new=max(lens))
    want_mem = memory.clone()
    want = kernel_refs.delta_rule(x, taps, x[:, C:], z.repeat_interleave(dim, 1) if head_decay else z,
                                  dt_bias.repeat_interleave(dim) if head_decay else dt_bias, a_log, torch.tensor(seq), torch.tensor(cu),
                                  torch.tensor(slots), want_mem, H, G, dim, vdim, dim ** -0.5, 1e-6)
    assert float((got.cpu() - want).abs().max()) < 3 * TOL * (1 + float(want.abs().max()))
    assert float((gm.cpu() - want_mem).abs().max()) < 3 * TOL * (1 + float(want_mem.abs().max()))


def test_preparation_places_and_taps(monkeypatch):
    """Runs of four tokens that begin at every place of a sequence, one sequence without a slot among them, and taps that are not 16-byte aligned: the
    same bits as each sequence alone (whose runs begin elsewhere) with aligned taps."""
    from dotllm_b200.kernels import ops
    monkeypatch.setattr(ops, "CHUNK_MIN_TOKENS", 2)
    H, G, dim, vdim, K = 4, 4, 64, 128, 4
    lens = [5, 6, 7, 9, 70, 3, 12, 33]
    C, T, n_state = 2 * G * dim + H * vdim, sum(lens), H * dim * vdim
    taps = g64(C, K, seed=1, scale=0.5).to(torch.bfloat16).to(DEV)
    odd = torch.empty(C * K + 1, dtype=torch.bfloat16, device=DEV)[1:].view(C, K).copy_(taps)
    assert taps.data_ptr() % 16 == 0 and odd.data_ptr() % 16 != 0
    dt_bias, a_log = g64(H * dim, seed=2).float().to(DEV), g64(H, seed=3, scale=0.5).float().to(DEV)
    x, z = g64(T, C + H, seed=10).to(torch.bfloat16).to(DEV), g64(T, H * dim, seed=20).float().to(DEV)
    memory = g64(9, n_state + (K - 1) * C, seed=4).float().to(DEV)
    slots = [4, 1, -1, 5, 0, 2, 8, 7]

    def run(rows, w, lengths, where):
        m = memory.clone()
        seq, cu = [i for i, n in enumerate(lengths) for _ in range(n)], [0] + list(np.cumsum(lengths))
        o = ops.delta_rule(x[rows], w, x[rows][:, C:], z[rows], dt_bias, a_log, i32(seq), i32(cu), i32(where), m, H, G, dim, vdim, dim ** -0.5, 1e-6,
                           max_new=max(lengths))
        return o, m

    whole, mem = run(slice(0, T), odd, lens, slots)
    at = 0
    for n, slot in zip(lens, slots):
        if slot >= 0:
            alone, m = run(slice(at, at + n), taps, [n], [slot])
            assert torch.equal(whole[at:at + n], alone) and torch.equal(mem[slot], m[slot])
        at += n
    assert torch.equal(mem[[3, 6]], memory[[3, 6]])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vdim,gate", [(128, "silu"), (64, "sigmoid"), (20, "silu")])
def test_head_norm_of_many_rows(dtype, vdim, gate):
    """So many (token, head) pairs that a warp takes four, not a multiple of a block's sixteen; the gate is a column view of wider rows."""
    from dotllm_b200.kernels import ops
    H, T = 7, 1361
    assert H * T % 16 and H * T >= 4 * 4 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    o, wide = g64(T, H * vdim, seed=1).float().to(DEV), g64(T, H * vdim + 8, seed=2).to(dtype).to(DEV)
    g, gain = wide[:, 8:], g64(vdim, seed=3).float().to(DEV)
    got = ops.head_norm_gate(o, g, gain, H, vdim, 1e-5, dtype, gate=gate)
    od, gd = o.double().view(T, H, vdim), g.double().reshape(T, H, vdim)
    want = od / (od.square().mean(-1, keepdim=True) + 1e-5).sqrt() * gain.double() * (torch.sigmoid(gd) * (gd if gate == "silu" else 1))
    # float32: a sum of 128 squares and a handful of roundings; bfloat16: the result's own rounding
    rel = 2e-6 if dtype == torch.float32 else 2.0 ** -8
    assert bool(((got.double().view(T, H, vdim) - want).abs() <= rel * want.abs() + 1e-6).all())
    few = ops.head_norm_gate(o[:3], g[:3], gain, H, vdim, 1e-5, dtype, gate=gate)          # a pair a warp: the same bits
    assert torch.equal(few, got[:3])
