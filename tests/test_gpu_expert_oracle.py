"""The expert forward against the oracle: groups and batches of slots that are full and ragged, columns that no block divides,
one slot, more slots than a warp has lanes, duplicates inside a token, empty and out-of-range slots."""

import pytest
import torch

from oracle import flashmoe_oracle as O

pytestmark = pytest.mark.gpu

BF, HF = torch.bfloat16, torch.float16


# tokens, hidden, experts, slots per token
@pytest.mark.parametrize(
    "T,H,N,k,dtype,seed,bad,zipf",
    [(64, 256, 512, 8, BF, 100, False, False), (200, 1024, 2048, 64, BF, 101, False, False),
     (96, 512, 1000, 20, BF, 102, False, False), (130, 1000, 777, 70, BF, 103, False, False),
     (77, 200, 300, 1, BF, 104, False, False), (128, 2048, 4096, 16, BF, 105, False, False),
     (150, 1536, 999, 130, HF, 106, False, False), (64, 64, 128, 33, HF, 107, False, False),
     (90, 768, 500, 24, BF, 300, True, False), (100, 1024, 64, 48, BF, 301, False, True)],
)
def test_expert_forward_matches_oracle(T, H, N, k, dtype, seed, bad, zipf):
    from flash_moe_b200 import _lib
    from flash_moe_b200.ops.flash_expert import _expert_forward

    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(T, H, generator=g) * 0.5).to(dtype)
    down = (torch.randn(N, H, generator=g) * 0.1).to(dtype)
    up = (torch.randn(N, H, generator=g) * 0.1).to(dtype)
    if zipf:  # many duplicates inside a token: they must accumulate
        p = torch.arange(1, N + 1, dtype=torch.float64).pow(-1.3)
        idx = torch.multinomial((p / p.sum()).float(), T * k, replacement=True, generator=g).view(T, k)
    else:
        idx = torch.randint(0, N, (T, k), generator=g)
    gates = torch.softmax(torch.randn(T, k, generator=g), -1).to(dtype)
    if bad:
        idx[0, 0] = -1          # empty slot: skipped silently
        idx[1, k - 1] = N + 5   # out of range: skipped and flagged
        idx[2, 0] = -7
    valid = (idx >= 0) & (idx < N)
    want = O.expert_forward(x.float(), down.float(), up.float(), idx.clamp(0, N - 1),
                            torch.where(valid, gates.float(), torch.zeros(())))
    args = [t.cuda() for t in (x, down, up, idx, gates)]
    got32 = _expert_forward(*args, out_dtype=torch.float32)
    got16, raw = _expert_forward(*args, save_scores=True)
    again = _expert_forward(*args, out_dtype=torch.float32)
    assert _lib.read_status() == (_lib.STATUS_BAD_EXPERT_ID if bad else 0)
    assert torch.equal(got32, again), "reruns must be bit-equal"
    assert float((got32.cpu() - want).abs().max() / want.pow(2).mean().sqrt()) < 2e-4
    O.assert_output_parity(got16.cpu(), want, dtype)
    s_want = (x.float()[:, None, :] * down.float()[idx.clamp(0, N - 1)]).sum(-1)
    s_want = torch.where(valid, s_want, torch.zeros(()))
    assert float((raw.cpu() - s_want).abs().max()) < 1e-3 * max(1.0, float(s_want.abs().max()))
