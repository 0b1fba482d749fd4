"""Linear attention with a decay per head in tiles of 64 tokens, where it can go wrong: chunks of one, several and a part of
a tile, rows just below, at and above a tile, key and value sizes that leave parts of a tile empty, decays of zero and one,
a state that is not zero, and rows that are no whole 16-byte pieces."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [64, 128, 256, 48])
@pytest.mark.parametrize("H,d,dv,lens,dtype,planes", [
    (2, 128, 128, [63, 64, 65, 1, 200], "bfloat16", 1), (2, 64, 200, [129, 255, 257], "bfloat16", 1),
    (3, 72, 40, [130, 0, 191], "bfloat16", 1), (2, 36, 70, [70, 128], "bfloat16", 1), (2, 128, 64, [300], "float32", 2),
    (2, 8, 8, [193], "bfloat16", 1), (2, 72, 136, [140, 66], "float32", 1), (3, 40, 20, [129], "float32", 3)])
def test_tiles_of_tokens_against_the_recurrence(H, d, dv, lens, dtype, planes, chunk):
    from kindi_b200.kernels import lib as K
    K.load()
    g = torch.Generator(device="cuda").manual_seed(H * d + dv + chunk)
    tdt = getattr(torch, dtype)
    B, T, ncol = len(lens), sum(lens), 2 * H * d + H * dv
    x = torch.randn(T, ncol, device="cuda", generator=g)
    if planes == 1:
        src = x.to(tdt)
        x = src
    else:
        src = torch.stack([x * 0.25, x * 0.75])
    decay = torch.tensor([0.0, 1.0, 0.97][:H], device="cuda") if H == 3 else torch.tensor([1.0, 0.9], device="cuda")
    slots = torch.tensor([(3 * b + 1) % (B + 3) for b in range(B)] if B != 3 else [2, 0, 4], dtype=torch.int32, device="cuda")
    state = torch.randn(B + 3, H, dv, d, device="cuda", generator=g)
    before = state.clone()
    q_start = torch.tensor([sum(lens[:b]) for b in range(B + 1)], dtype=torch.int32, device="cuda")
    out = torch.full((T, H * dv), float("nan"), device="cuda")
    K.decay_scan(src, B, H, d, dv, decay, q_start, slots, state, out, chunk=chunk, max_rows=max(lens) + 3)
    xd = torch.nn.functional.silu(x.double())
    q, k, v = xd[:, :H * d].view(T, H, d), xd[:, H * d:2 * H * d].view(T, H, d), xd[:, 2 * H * d:].view(T, H, dv)
    untouched = set(range(B + 3)) - set(slots.tolist())
    for s in untouched:
        assert torch.equal(state[s], before[s])
    for b, n in enumerate(lens):
        S = before[int(slots[b])].double().transpose(1, 2)
        size = S.abs()                                # what the terms add up to without their signs
        for t in range(sum(lens[:b]), sum(lens[:b]) + n):
            kv = k[t][:, :, None] * v[t][:, None, :]
            S, size = decay.double()[:, None, None] * S + kv, decay.double()[:, None, None] * size + kv.abs()
            want, most = torch.einsum("hde,hd->he", S, q[t]), torch.einsum("hde,hd->he", size, q[t].abs())
            # 32-bit sums of up to n + d terms, rounded silu (2^-21) in every factor: far below 1e-5 of the terms' sum
            assert float(((out[t].view(H, dv).double() - want).abs() / (most + 1e-30)).max()) < 1e-5, (b, t)
        assert float(((state[int(slots[b])].double().transpose(1, 2) - S).abs() / (size + 1e-30)).max()) < 1e-5, b


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("dtype,chunk", [("bfloat16", 64), ("bfloat16", 128), ("float32", 64), ("bfloat16", 48)])
def test_what_is_not_finite_stays_out_of_earlier_tokens(dtype, chunk, bad):
    """a value, key or query that is no number or infinite changes no earlier token, and a value no other column"""
    from kindi_b200.kernels import lib as K
    K.load()
    H, d, dv, T = 2, 64, 72, 150
    g = torch.Generator(device="cuda").manual_seed(chunk)
    clean = torch.randn(T, 2 * H * d + H * dv, device="cuda", generator=g).to(getattr(torch, dtype))
    decay = torch.tensor([1.0, 0.95], device="cuda")
    q_start = torch.tensor([0, T], dtype=torch.int32, device="cuda")
    state0 = torch.randn(1, H, dv, d, device="cuda", generator=g)

    def go(x):
        out = torch.full((T, H * dv), float("nan"), device="cuda")
        K.decay_scan(x, 1, H, d, dv, decay, q_start, torch.zeros(1, dtype=torch.int32, device="cuda"), state0.clone(), out,
                     chunk=chunk, max_rows=T)
        return out.view(T, H, dv)
    want = go(clean)
    assert bool(want.isfinite().all())
    for s in (1, 15, 16, 37, 63, 64, 79, 127, T - 1):
        for kind, col in (("v", 2 * H * d + 5), ("v", 2 * H * d + dv + 70), ("k", H * d + 3), ("q", d + 1)):
            x = clean.clone()
            x[s, col] = bad
            got = go(x)
            h = {"v": (col - 2 * H * d) // dv, "k": (col - H * d) // d, "q": col // d}[kind]
            assert torch.equal(got[:s], want[:s]), (kind, s)
            assert torch.equal(got[:, 1 - h], want[:, 1 - h]), (kind, s)
            if kind == "v":
                e = (col - 2 * H * d) % dv
                others = [c for c in range(dv) if c != e]
                assert torch.equal(got[:, :, others], want[:, :, others]), s
            if kind == "q":
                assert torch.equal(got[s + 1:], want[s + 1:]), s


@pytest.mark.parametrize("d,chunk,max_rows", [(8, 41000, 300), (128, 32448, 300), (128, 32449, 300), (72, 45000, 100000), (8, 65, 33000 * 65),
                                              (8, 128, 32767 * 128)])
def test_chunks_of_any_length_and_number(d, chunk, max_rows):
    """chunks whose powers of the decay do not fit the tiles' shared memory, and more tiles than their grid takes"""
    from kindi_b200.kernels import lib as K
    K.load()
    H, dv, lens = 1, 8, [130, 1]
    g = torch.Generator(device="cuda").manual_seed(d)
    x = torch.randn(sum(lens), 2 * H * d + H * dv, device="cuda", generator=g).to(torch.bfloat16)
    decay, slots = torch.tensor([0.97], device="cuda"), torch.tensor([1, 0], dtype=torch.int32, device="cuda")
    q_start = torch.tensor([0, 130, 131], dtype=torch.int32, device="cuda")
    state0 = torch.randn(2, H, dv, d, device="cuda", generator=g)
    got = []
    for more in (dict(), dict(chunk=chunk, max_rows=max_rows)):
        state, out = state0.clone(), torch.full((sum(lens), H * dv), float("nan"), device="cuda")
        K.decay_scan(x, 2, H, d, dv, decay, q_start, slots, state, out, **more)
        got.append((out, state))
    for a, b in zip(*got):
        # (the token-by-token form, whose sums are taken in another order)
        assert float((a - b).abs().max() / a.abs().max()) < 1e-5


@pytest.mark.parametrize("d,copies", [(128, 0), (129, 1)])
def test_scratch_is_what_the_form_reads(d, copies):
    from kindi_b200.kernels import lib as K
    K.load()
    B, H, dv, n, chunk = 4, 8, 256, 60, 64
    x = torch.randn(B * n, 2 * H * d + H * dv, device="cuda").to(torch.bfloat16)
    q_start = torch.arange(B + 1, dtype=torch.int32, device="cuda") * n
    slot = torch.arange(B, dtype=torch.int32, device="cuda")
    state, out = torch.zeros(B, H, dv, d, device="cuda"), torch.empty(B * n, H * dv, device="cuda")
    decay = torch.full((H,), 0.9, device="cuda")
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    K.decay_scan(x, B, H, d, dv, decay, q_start, slot, state, out, chunk=chunk, max_rows=n)
    used = torch.cuda.max_memory_allocated() - before
    assert state.nbytes * (1 + copies) <= used < state.nbytes * (1.5 + copies)
