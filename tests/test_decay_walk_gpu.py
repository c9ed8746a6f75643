"""The walk of long portions with 64 key channels against the stand-in of the same name: portions
that end inside, on and behind a batch of 16 tokens and a segment of 128, single tokens beside them, both decays, both
numbers of value columns, states that a step before left, and column ranges that only the general
kernel takes."""

import pytest
import torch

import fake_kernels as fake
from test_kernels_gpu import close, make_step, ops, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", ["channel", "head"])
@pytest.mark.parametrize("vdim,lead,rotary", [(64, 0, 64), (128, 4, 16), (64, 3, 64), (192, 0, 0)])
@pytest.mark.parametrize("q_lens", [[64, 1, 80], [15, 97], [128, 129], [1, 700, 3], [256]])
def test_walk_of_long_portions(dtype, kind, vdim, lead, rotary, q_lens):
    heads, dim, t = 3, 64, ops()
    starts = [7 * s for s in range(len(q_lens))]
    cpu, gpu, _ = make_step(q_lens, starts, 16, 64, 3, num_slots=5)
    gpu.all_decode, gpu.max_q_len = False, max(q_lens)
    rows, qk, vg = sum(q_lens), heads * dim, heads * vdim
    x = rnd((rows, lead + 2 * qk + 2 * vg), dtype, 1, 0.5)
    parts = lambda y: [y[:, lead + a : lead + b] for a, b in ((0, qk), (qk, 2 * qk), (2 * qk, 2 * qk + vg), (2 * qk + vg, 2 * qk + 2 * vg))]
    state = rnd((5, heads, dim, vdim), torch.float32, 2, 0.1)
    if kind == "channel":
        kw = {"decay_logits": rnd((rows, qk), torch.float32, 3, 0.5), "decay_bias": rnd((qk,), torch.float32, 4) - 2.0,
              "bonus": rnd((heads, dim), torch.float32, 5, 0.3) + 0.5}
    else:
        decay = torch.tensor([0.96875, 0.998, 0.5])
        kw = {"head_decay": decay, "inv_freq": 10000.0 ** (-torch.arange(0, rotary, 2, dtype=torch.float32) / max(1, rotary)),
              "rotary_dim": rotary, "key_scale": 0.125}
    kw["out_weight"] = rnd((vg,), torch.float32, 6) + 1.0
    want, want_state = torch.zeros(rows, vg, dtype=dtype), state.clone()
    q, k, v, gate = parts(x)
    fake.decay_recurrence(q, k, v, want, want_state, cpu, heads, dim, vdim, 1e-5, gate=gate, out_scale=0.5, **kw)
    got, got_state = torch.zeros(rows, lead + vg, dtype=dtype).cuda(), state.cuda()
    q, k, v, gate = parts(x.cuda())
    on_gpu = {n: (y.cuda() if torch.is_tensor(y) else y) for n, y in kw.items()}
    t.decay_recurrence(q, k, v, got[:, lead:], got_state, gpu, heads, dim, vdim, 1e-5, gate=gate, out_scale=0.5, **on_gpu)
    # (float32 sums over at most 700 tokens of 64 channels: the bound of the general kernel's tests)
    close(got[:, lead:], want, dtype, f"walk {kind} {vdim} {q_lens}", rel32=2e-5)
    close(got_state, want_state, torch.float32, f"state {kind} {vdim} {q_lens}", rel32=2e-5)
