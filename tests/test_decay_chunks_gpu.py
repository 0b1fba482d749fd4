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
    (2, 8, 8, [193], "bfloat16", 1)])
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
