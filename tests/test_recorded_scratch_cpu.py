"""What a recorded step was given stays as it is while larger steps come: the scratch of products whose tiles two pairs of SMs
finish together, and the weights of one."""
import torch

from kindi_b200.kernels import fast


def test_scratch_of_a_recorded_step_is_never_handed_on(monkeypatch):
    monkeypatch.setattr(fast, "_PAIR_SCRATCH", {})
    monkeypatch.setattr(fast, "_PAIR_RETIRED", [])
    dev = torch.device("cpu")
    small = fast._pair_scratch(dev, 2, 64, False)
    assert fast._pair_scratch(dev, 1, 64, True) is small                  # (a recording takes what is there)
    own = fast._pair_scratch(dev, 5, 64, True)                            # (or gets one of its own)
    assert own is not small and fast._PAIR_SCRATCH[dev] is small and int(own[1].abs().sum()) == 0
    large = fast._pair_scratch(dev, 3, 64, False)
    assert large[0].numel() >= 2 * small[0].numel() and large[1].numel() >= 2 * small[1].numel()
    assert fast._PAIR_SCRATCH[dev] is large and any(s is small for s in fast._PAIR_RETIRED)
    for part, flags in (small, large):
        flags.fill_(1)
    fast.reset_scratch()                                                  # (after an error: those of recorded steps, too)
    assert int(small[1].sum()) == 0 and int(large[1].sum()) == 0


def test_weights_of_one_outlive_many_sizes(monkeypatch):
    monkeypatch.setattr(fast, "_ONES", {})
    first = fast._ones_like(torch.empty(7, 2))
    for n in range(1, 300):
        assert torch.equal(fast._ones_like(torch.empty(n)), torch.ones(n))
    kept = fast._ONES[torch.device("cpu")]
    assert first.data_ptr() == kept[0].data_ptr() and len(kept) < 10 and torch.equal(first, torch.ones(14))
