"""The stages of the fused chunk kernel: chunk counts around its rings of gate and q / k tiles, repeatability over fresh
buffers (a tile refilled before its last reader shows here first), inputs of the least alignment that the call takes."""
import random

import pytest
import torch

import kda_oracle as ko
from kda_testlib import DEV, D, cu_of, gold_plain, gold_raw, plain_on_device, to_dev

pytestmark = pytest.mark.gpu

# one to eight chunks, full and partial: the q / k ring has two or three stages, its barriers repeat after six chunks
LENS = [1, 31, 32, 33, 64, 65, 96, 97, 128, 159, 161, 192, 223, 225, 256]


@pytest.fixture(scope="module")
def kda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import kda_b200
    from kda_b200 import _cabi
    _cabi.lib()
    return kda_b200


@pytest.mark.parametrize("order", [1, -1])
def test_chunk_counts_raw(kda, order):
    lens = LENS[::order]
    inputs = ko.make_inputs_raw(2, lens, 31)
    gold_o, gold_s, _ = gold_raw(inputs, lens)
    out, fin = kda.run(*to_dev(inputs))
    torch.cuda.synchronize()
    ko.check_close(out.cpu(), gold_o, "output")
    ko.check_close(fin.cpu(), gold_s, "final state")


@pytest.mark.parametrize("g_mean", [0.0, 4.0])
def test_chunk_counts_plain(kda, g_mean):
    lens, H = LENS, 2
    q, k, v, g, beta = plain_on_device(H, sum(lens), 32, g_mean)
    init = torch.randn(len(lens), H, D, D, generator=torch.Generator(device=DEV).manual_seed(33), device=DEV) * 0.05
    out, fin = kda.chunk_kda(q, k, v, g, beta, initial_state=init, output_final_state=True, cu_seqlens=cu_of(lens))
    torch.cuda.synchronize()
    gold_o, gold_s, _ = gold_plain(q.cpu(), k.cpu(), v.cpu(), g.cpu(), beta.cpu(), D ** -0.5, init.cpu(), lens)
    ko.check_close(out.cpu(), gold_o, "output")
    ko.check_close(fin.cpu(), gold_s, "final state")


@pytest.mark.parametrize("raw", [True, False])
def test_repeatable_over_fresh_buffers(kda, raw):
    """About seven hundred ragged (sequence, head) tasks, five times over new tensors: the same bits."""
    rng, H = random.Random(5), 32
    lens = [rng.randint(1, 900) for _ in range(22)]
    first = None
    for _ in range(5):
        q, k, v, g, beta = plain_on_device(H, sum(lens), 34)
        init = torch.randn(len(lens), H, D, D, generator=torch.Generator(device=DEV).manual_seed(35), device=DEV) * 0.05
        if raw:
            res = kda.kda_prefill(q, k, v, g.to(torch.bfloat16), beta.to(torch.bfloat16), torch.zeros(H, device=DEV),
                                  torch.zeros(H * D, device=DEV), init, cu_of(lens))
        else:
            res = kda.chunk_kda(q, k, v, g, beta, initial_state=init, output_final_state=True, cu_seqlens=cu_of(lens))
        torch.cuda.synchronize()
        res = [t.clone() for t in res]
        if first is None:
            first = res
        assert all(torch.equal(a, b) for a, b in zip(res, first))


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_dt_bias_of_any_alignment(kda, offset):
    H, lens = 2, [70, 33]
    inputs = to_dev(ko.make_inputs_raw(H, lens, 36))
    ref = kda.run(*inputs)
    buf = torch.empty(H * D + 4, device=DEV)
    dt = buf[offset:offset + H * D]
    dt.copy_(inputs[6])
    inputs[6] = dt
    res = kda.run(*inputs)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(res, ref))


@pytest.mark.parametrize("raw", [True, False])
def test_a_head_alone_and_among_all(kda, raw):
    """Every SM busy against a handful of CTAs: a tile handed back to the copy engine before its last read would show as
    different bits.  Heads are independent, and uncut runs do the same arithmetic in both launches."""
    H, lens = 48, [1500, 37, 700, 64, 333, 1024]
    q, k, v, g, beta = plain_on_device(H, sum(lens), 41)
    init = torch.randn(len(lens), H, D, D, generator=torch.Generator(device=DEV).manual_seed(42), device=DEV) * 0.05
    if raw:
        g, beta = g.to(torch.bfloat16), beta.to(torch.bfloat16)
    A_log, dt_bias = torch.zeros(H, device=DEV), torch.zeros(H * D, device=DEV)

    def call(lo, hi):
        t = [x[:, :, lo:hi] for x in (q, k, v, g, beta)]
        s0 = init[:, lo:hi].contiguous()
        if raw:
            launch = kda.prepare(*t, A_log[lo:hi], dt_bias[lo * D:hi * D], D ** -0.5, s0, cu_of(lens), max_cut_pieces=0)
        else:
            launch = kda.prepare_plain(*t, initial_state=s0, output_final_state=True, cu_seqlens=cu_of(lens), max_cut_pieces=0)
        return launch()

    out, fin = call(0, H)
    for h in (0, 17, H - 1):
        o, f = call(h, h + 1)
        torch.cuda.synchronize()
        assert torch.equal(o[:, :, 0], out[:, :, h]) and torch.equal(f[:, 0], fin[:, h])


def _rows_before(kda, token, value):
    """Rows in front of `token`, whose gates are `value` in every channel: the output, the fp64 recurrence, the status."""
    H, T = 2, 90
    q, k, v, g, beta = plain_on_device(H, T, 51, 3.0)
    init = torch.randn(1, H, D, D, generator=torch.Generator(device=DEV).manual_seed(52), device=DEV) * 0.05
    cut = [t[:, :token].cpu() for t in (q, k, v, g, beta)]
    g[:, token] = value
    launch = kda.prepare_plain(q, k, v, g, beta, initial_state=init, output_final_state=True)
    out, _ = launch()
    torch.cuda.synchronize()
    gold, _, _ = gold_plain(*cut, D ** -0.5, init.cpu(), [token])
    return out[:, :token].float().cpu(), gold, kda.status_bits(launch)


@pytest.mark.parametrize("value", [-90.0, -1400.0, -1500.0, -1e9, float("-inf")])
@pytest.mark.parametrize("token", [16, 19, 22, 27, 31, 32 + 21, 64 + 25])
def test_rows_in_front_of_a_reset_keep_their_decay(kda, token, value):
    """One token of a chunk's second half decays without bound (a state reset): the chunk is reported as out of range, and
    the tokens in front of that one do not depend on its gates."""
    out, gold, status = _rows_before(kda, token, value)
    assert status == 16
    ko.check_close(out, gold, f"rows in front of token {token}")


@pytest.mark.parametrize("token", [16, 19, 27, 31, 32 + 21, 64 + 25])
def test_rows_in_front_of_a_gate_that_is_not_a_number(kda, token):
    """A NaN gate in a chunk's second half reaches its own token and what follows, not the rows in front of it."""
    out, gold, status = _rows_before(kda, token, float("nan"))
    assert status == 0
    ko.check_close(out, gold, f"rows in front of token {token}")


@pytest.mark.parametrize("token", [16, 19, 27, 31, 32 + 21, 64 + 25])
def test_rows_in_front_of_a_raw_gate_that_is_not_a_number(kda, token):
    inputs = ko.make_inputs_raw(2, [90], 53)
    gold, _, _ = gold_raw([t[:, :token] for t in inputs[:5]] + list(inputs[5:9]), [token])
    inputs[3][:, token] = float("nan")
    out, _ = kda.run(*to_dev(inputs))
    torch.cuda.synchronize()
    ko.check_close(out[:, :token].float().cpu(), gold, f"rows in front of token {token}")


@pytest.mark.parametrize("raw", [True, False])
def test_strided_tokens_of_the_least_alignment(kda, raw):
    """q, k, v, g as slices whose base and token stride are multiples of 16 bytes and of nothing more: read in place."""
    H, lens = 3, [70, 1, 161]
    T = sum(lens)
    q, k, v, g, beta = plain_on_device(H, T, 71)
    if raw:
        g, beta = g.to(torch.bfloat16), beta.to(torch.bfloat16)
    A_log, dt_bias = torch.zeros(H, device=DEV), torch.zeros(H * D, device=DEV)
    init = torch.randn(len(lens), H, D, D, generator=torch.Generator(device=DEV).manual_seed(72), device=DEV) * 0.05

    def sliced(t):
        pad = 16 // t.element_size() if t.element_size() == 2 else 8     # (the token stride: a multiple of eight elements)
        wide = torch.full((T, H * D + 3 * pad), float("nan"), dtype=t.dtype, device=DEV)
        part = wide[:, 16 // t.element_size():][:, :H * D]
        part.copy_(t.view(T, H * D))
        return part.unflatten(1, (H, D))[None]

    def launch(t):
        if raw:
            return kda.prepare(*t, beta, A_log, dt_bias, D ** -0.5, init, cu_of(lens))
        return kda.prepare_plain(*t, beta, initial_state=init, output_final_state=True, cu_seqlens=cu_of(lens))

    views = [sliced(t) for t in (q, k, v, g)]
    assert all(t.data_ptr() % 32 == 16 for t in views)
    there, here = launch(views), launch([q, k, v, g])
    assert there._copies == []
    a, b = there(), here()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(a, b))
