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


# Any cut, any neighbours and either kernel: the same bits.


class Portions:
    """One sequence's rows (or several) and what the recurrence makes of them, however they are cut."""

    def __init__(self, kind, vdim, dtype, rows, lead=0, rotary=64, extremes=False, heads=3):
        self.kind, self.vdim, self.dtype, self.lead, self.heads, self.rotary = kind, vdim, dtype, lead, heads, rotary
        qk, vg = heads * 64, heads * vdim
        x = torch.zeros(rows, lead + 2 * qk + 2 * vg, dtype=dtype)
        x[:, lead:] = rnd((rows, 2 * qk + 2 * vg), dtype, 1, 0.5)
        self.x = x.cuda()
        if kind == "channel":
            logits, bias = rnd((rows, qk), torch.float32, 3, 0.5), rnd((qk,), torch.float32, 4) - 2.0
            if extremes:  # w = 1 for the even channels, w = 0 for every third of the others at single tokens
                bias[::2] = -200.0
                logits[120:140:3, 1::3] = 60.0
            self.kw = {"decay_logits": logits.cuda(), "decay_bias": bias.cuda(), "bonus": (rnd((heads, 64), torch.float32, 5, 0.3) + 0.5).cuda()}
        else:
            loss = torch.tensor([0.0, 1.0, 0.015625] if extremes else [0.03125, 0.002, 0.5])[torch.arange(heads) % 3]
            self.kw = {"head_decay": (1.0 - loss).cuda(), "head_loss": loss.cuda(), "rotary_dim": rotary, "key_scale": 0.125,
                       "inv_freq": (10000.0 ** (-torch.arange(0, rotary, 2, dtype=torch.float32) / max(1, rotary))).cuda()}
        self.kw["out_weight"] = (rnd((vg,), torch.float32, 6) + 1.0).cuda()
        self.state = rnd((12, heads, 64, vdim), torch.float32, 2, 0.1).cuda()

    def step(self, first, q_lens, starts, slots, hint=None):
        """A step of the rows from `first` on; the outputs."""
        t, qk, vg = ops(), self.heads * 64, self.heads * self.vdim
        rows = slice(first, first + sum(q_lens))
        _, gpu, _ = make_step(q_lens, starts, 16, 256, 3)
        gpu.state_slots = torch.tensor(slots, dtype=torch.int32).cuda()
        gpu.all_decode, gpu.max_q_len = max(q_lens) == 1, hint or max(q_lens)
        x = self.x[rows, self.lead :]
        part = lambda a, n: x[:, a : a + n]
        kw = dict(self.kw)
        if self.kind == "channel":
            kw["decay_logits"] = kw["decay_logits"][rows].contiguous()
        out = torch.zeros(sum(q_lens), self.lead + vg, dtype=self.dtype, device="cuda")[:, self.lead :]
        t.decay_recurrence(part(0, qk), part(qk, qk), part(2 * qk, vg), out, self.state, gpu, self.heads, 64, self.vdim, 1e-5,
                           gate=part(2 * qk + vg, vg), out_scale=0.5, **kw)
        return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind,vdim", [("channel", 64), ("channel", 128), ("head", 64), ("head", 128)])
@pytest.mark.parametrize("extremes", [False, True])
def test_cuts_and_neighbours_change_no_bit(dtype, kind, vdim, extremes):
    rows = 700
    whole = Portions(kind, vdim, dtype, rows, extremes=extremes)
    want = whole.step(0, [rows], [0], [4])
    for cut in ([300, 1, 399], [128, 572], [64] * 10 + [60], [257, 20, 20, 3, 400]):
        pieces, got, at = Portions(kind, vdim, dtype, rows, extremes=extremes), [], 0
        for n in cut:
            got.append(pieces.step(at, [n], [at], [4]))
            at += n
        assert torch.equal(pieces.state[4], whole.state[4]), cut
        got = torch.cat(got)
        if min(cut) >= 64:  # (the row kernel's unit RMS throughout)
            assert torch.equal(got, want), cut
        else:  # short portions: other orders of the squares' sum, and with 128 value columns of a column's (the bound above)
            close(got, want, dtype, f"outputs {cut}", rel32=2e-5)
    # the same rows as the second of five sequences, two of them without rows, and two single tokens behind
    beside = Portions(kind, vdim, dtype, rows, extremes=extremes)
    beside.x, before = torch.cat([beside.x[:150], beside.x, beside.x[:2]]), beside.state.clone()
    if kind == "channel":
        z = beside.kw["decay_logits"]
        beside.kw["decay_logits"] = torch.cat([z[:150], z, z[:2]])
    # (positions start with each sequence, the rotation's as well)
    got = beside.step(0, [150, 0, rows, 0, 1, 1], [0, 0, 0, 0, 0, 0], [3, 5, 4, 6, 0, 1])
    assert torch.equal(got[150 : 150 + rows], want) and torch.equal(beside.state[4], whole.state[4])
    for untouched in (2, 5, 6, 7, 11):
        assert torch.equal(beside.state[untouched], before[untouched])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind,vdim,rotary", [("channel", 64, 0), ("channel", 128, 0), ("head", 64, 64), ("head", 128, 16), ("head", 192, 20)])
def test_walk_and_general_kernel_give_the_same_bits(dtype, kind, vdim, rotary):
    """Rows on no 8-byte boundary (and a rotation over no multiple of eight channels) take the general
    kernel, with the same number of lanes to a column."""
    q_lens, starts, slots = [90, 300, 1, 130], [5, 0, 40, 17], [3, 0, 7, 2]
    walk, general = (Portions(kind, vdim, dtype, sum(q_lens), lead, rotary, heads=4) for lead in (0, 3))
    a, b = walk.step(0, q_lens, starts, slots), general.step(0, q_lens, starts, slots)
    assert torch.equal(walk.state, general.state)
    assert torch.equal(a, b)


@pytest.mark.parametrize("kind,vdim", [("channel", 64), ("head", 128)])
@pytest.mark.parametrize("hint", [64, 127, 128, 129])
def test_a_longest_portion_that_is_wrong_costs_no_bit(kind, vdim, hint):
    """What a step says its longest portion is chooses a route: a captured step says the same for many."""
    q_lens, starts, slots = [300, 1, 200], [0, 9, 30], [4, 2, 9]
    right, wrong = (Portions(kind, vdim, torch.bfloat16, sum(q_lens)) for _ in range(2))
    want, got = right.step(0, q_lens, starts, slots), wrong.step(0, q_lens, starts, slots, hint=hint)
    assert torch.equal(got, want) and torch.equal(wrong.state, right.state)


@pytest.mark.parametrize("vdim,lead,q_lens,what", [
    (64, 3, [300], "(columns over 8 CTAs)"), (128, 3, [300], "(columns over 8 CTAs)"), (64, 0, [30, 40], "decay_recurrence"),
])
def test_what_the_walk_does_not_take_shares_its_columns_out(monkeypatch, vdim, lead, q_lens, what):
    seen = launches_of(monkeypatch, lambda: Portions("head", vdim, torch.bfloat16, sum(q_lens), lead).step(
        0, q_lens, [0] * len(q_lens), list(range(len(q_lens)))))
    assert len(seen) == 1 and seen[0][0].endswith(what), seen


def launches_of(monkeypatch, call):
    """(what, launches) of every entry of the launch table that a call makes."""
    from shiso_llm_b200.kernels import ops as table

    seen, done = [], table._done
    monkeypatch.setattr(table, "_done", lambda status, name, count=1, shape=(): (seen.append((name, count)), done(status, name, count, shape)))
    call()
    return seen


@pytest.mark.parametrize("vdim,lead,q_lens,what,launches", [
    (64, 0, [300], "(walk of segments)", 3), (128, 0, [300, 2], "(walk of segments)", 3), (64, 0, [100, 90], "(walk)", 2), (64, 3, [300], "(columns over 8 CTAs)", 2),
    (64, 0, [30, 40], "decay_recurrence", 1),
])
def test_a_recurrence_counts_its_launches(monkeypatch, vdim, lead, q_lens, what, launches):
    seen = launches_of(monkeypatch, lambda: Portions("head", vdim, torch.bfloat16, sum(q_lens), lead).step(
        0, q_lens, [0] * len(q_lens), list(range(len(q_lens)))))
    assert len(seen) == 1 and seen[0][0].endswith(what) and seen[0][1] == launches, seen
