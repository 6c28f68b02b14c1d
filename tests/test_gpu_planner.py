"""The device planner's table checks and task order at the sizes where it changes its method, against the fp64 oracle.

Short sequences on one head: what is tested is that every sequence is run exactly once, from its own state into its own
slot and checkpoint rows, whichever way the tables were checked and the tasks ordered."""
import random

import pytest
import torch

import kda_oracle as ko
from kda_testlib import DEV, D, cu_of, gold_raw, to_dev

pytestmark = pytest.mark.gpu


def _serving_call(lens, slots, P, seed, every=0, starts=None, rows=0):
    """One call on a pool of P slots; the outcome that the tables call for, in ascending order of the sequences: the
    first claim of a slot keeps it (a later one starts from zeros and its state is dropped), checkpoint rows that overlap
    rows an earlier sequence keeps are not written.  Returns (launch, sequences that keep their rows)."""
    import kda_b200
    N = len(lens)
    inputs = ko.make_inputs_raw(1, lens, seed)
    q, k, v, g, beta, A_log, dt_bias, scale = to_dev(inputs[:8])
    pool0 = torch.randn(P, 1, D, D, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV) * 0.25
    pool = pool0.clone()
    kw = dict(dynamic_layout=True, ssm_state_indices=torch.tensor(slots, dtype=torch.int32, device=DEV))
    if every:
        ck = torch.full((rows, 1, D, D), float("nan"), device=DEV)
        kw.update(state_checkpoints=ck, checkpoint_cu_starts=torch.tensor([*starts, 0], dtype=torch.int64, device=DEV),
                  checkpoint_every_n_tokens=every)
    launch = kda_b200.prepare(q, k, v, g, beta, A_log, dt_bias, scale, pool, cu_of(lens), **kw)
    out = launch()[0]
    torch.cuda.synchronize()
    tag = f"N={N} lens={lens[:6]} slots={slots[:6]}"

    claimed, keeps_slot = set(), []
    for s in slots:
        keeps_slot.append(s not in claimed)
        claimed.add(s)
    own = torch.tensor(keeps_slot)
    start = pool0[torch.tensor(slots, device=DEV)].cpu()
    start[~own] = 0.0
    gold_o, gold_s, gold_ck = gold_raw(inputs[:8], lens, init=start, every=every)
    ko.check_close(out.cpu(), gold_o, tag + " output")
    live = torch.tensor([s for s, ok in zip(slots, keeps_slot) if ok], device=DEV)
    ko.check_close(pool[live].cpu(), gold_s[own], tag + " pool slots")
    others = torch.ones(P, dtype=torch.bool, device=DEV)
    others[live] = False
    assert torch.equal(pool[others], pool0[others]), tag + ": other pool slots modified"

    kept, taken, at = [], set(), 0
    for n in range(N if every else 0):
        count = -(-lens[n] // every)
        mine = set(range(starts[n], starts[n] + count))
        if not mine & taken:
            kept.append(n)
            taken |= mine
            if count:
                ko.check_close(ck[starts[n]:starts[n] + count].cpu(), gold_ck[at:at + count], f"{tag} rows of sequence {n}")
        at += count
    if every:
        free = torch.tensor([r not in taken for r in range(rows)], device=DEV)
        assert bool(torch.isnan(ck[free]).all()), tag + ": rows of no sequence were written"
    bits = (0 if all(keeps_slot) else 2) | (8 if every and len(kept) < N else 0)
    assert kda_b200.status_bits(launch) == bits and kda_b200.kernel_error(launch) == 0, tag
    return launch, kept


def _short_lengths(N, rng):
    return [rng.choice([0, 1, 31, 32, 33]) if rng.random() < 0.2 else rng.randint(1, 12) for _ in range(N - 1)] + [70]


@pytest.mark.parametrize("repeat", [False, True])
@pytest.mark.parametrize("N", [1, 2, 5, 6, 384, 385, 512, 513, 1025, 2048, 2049, 4096, 4097])
def test_slots_and_order(N, repeat):
    rng = random.Random(N)
    lens = _short_lengths(N, rng)
    slots = rng.sample(range(N + 5), N)
    if repeat:
        slots[-1] = slots[N // 3]                # for one sequence: the same table again
    _serving_call(lens, slots, N + 5, 40 + N)


@pytest.mark.parametrize("lens,starts,kept", [
    ([100], [1], [0]), ([100, 33], [2, 0], [0, 1]), ([100, 33], [0, 3], [0]),
    ([100, 33, 0, 1, 64], [5, 3, 0, 2, 0], [0, 1, 2, 3, 4]), ([100, 33, 0, 1, 64], [0, 4, 0, 6, 5], [0, 1, 2, 3]),
    ([100, 33, 1, 64, 31, 32, 1], [0, 4, 6, 7, 9, 10, 11], [0, 1, 2, 3, 4, 5, 6]),         # ascending
    ([100, 33, 1, 64, 31, 32, 1], [8, 6, 5, 3, 2, 1, 0], [0, 1, 2, 3, 4, 5, 6]),           # descending
    ([100, 33, 0, 64, 0, 32, 0, 0], [0, 4, 6, 6, 0, 8, 0, 0], list(range(8))),             # empty sequences padded with 0
    ([100, 33, 1, 64, 31, 32, 1], [0, 4, 6, 7, 9, 10, 2], [0, 1, 2, 3, 4, 5]),             # the last one into the first's rows
    ([100, 33, 64, 64, 31, 32, 1], [0, 3, 4, 6, 8, 9, 10], [0, 2, 3, 4, 5, 6])])           # a rejected one blocks nobody
def test_checkpoint_tables(lens, starts, kept):
    """Checkpoint rows every 32 tokens: ranges that go down, holes, empty sequences at row 0, overlaps."""
    assert _serving_call(lens, random.Random(2).sample(range(9), len(lens)), 9, 60 + len(lens), 32, starts, 12)[1] == kept


def test_slots_with_one_hash_entry():
    """Slots whose first entry in the planner's hash set (4096 entries, Fibonacci hashing) is one of four neighbours
    around the end of the set: they probe one another's entries and wrap; one of them is repeated behind them all."""
    P = 16384
    slots = [d for d in range(P) if (d * 2654435761 % 2**32 >> 20) in (4094, 4095, 0, 1)]
    assert len(slots) > 8
    random.Random(5).shuffle(slots)
    lens = _short_lengths(len(slots), random.Random(6))
    _serving_call(lens, slots, P, 70)
    _serving_call(lens + [3], slots + [slots[1]], P, 71)


@pytest.mark.parametrize("N", [384, 385, 1024, 1025])
def test_cuts_follow_either_order(N):
    """One long sequence among many short ones is cut, whichever way the tasks were ordered (up to 1024 sequences)."""
    rng = random.Random(N)
    lens = [rng.randint(1, 8) for _ in range(N)]
    lens[N // 2] = 4096
    launch, _ = _serving_call(lens, rng.sample(range(N + 5), N), N + 5, 80)
    na, nb, cut = launch.plan_counts()
    assert cut == (1 if N <= 1024 else 0) and na + nb >= N, (na, nb, cut)
