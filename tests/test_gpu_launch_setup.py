"""What a launch object answers before its first launch, and what setting one up costs."""
import ctypes

import pytest
import torch

import kda_oracle as ko
from kda_testlib import DEV, plain_on_device, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import kda_b200
    from kda_b200 import _cabi
    _cabi.lib()
    return kda_b200


@pytest.mark.parametrize("n,pieces", [(1, 0), (1, 2), (48, 128), (6, 1), (513, 37)])
def test_counts_lie_in_the_part_to_clear(kda, n, pieces):
    """Everything behind the bytes that the library names may hold anything."""
    from kda_b200 import _cabi
    lib, H = _cabi.lib(), 2
    size, clear = lib.kda_prefill_workspace_bytes_cuts(n, H, pieces), lib.kda_prefill_workspace_clear_bytes()
    assert 12 <= clear <= size
    ws = torch.full((size,), 0xAB, dtype=torch.uint8, device=DEV)
    assert ws.data_ptr() % 256 == 0
    ws[:clear].zero_()
    a = _cabi.KdaPrefillArgs()
    a.H, a.N, a.max_cut_pieces, a.workspace, a.workspace_bytes = H, n, pieces, ws.data_ptr(), size
    counts = (ctypes.c_int32 * 3)(7, 7, 7)
    assert lib.kda_prefill_plan_counts(ctypes.byref(a), counts, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert tuple(counts) == (0, 0, 0)


@pytest.mark.parametrize("heads,lens", [(2, [40]), (4, [4096, 33]), (3, [5] * 70)])
def test_nothing_is_reported_before_the_first_launch(kda, heads, lens):
    """Also when the memory held something else before."""
    inputs = to_dev(ko.make_inputs_raw(heads, lens, 61))
    for _ in range(2):
        used = [torch.full((n,), 0xAB, dtype=torch.uint8, device=DEV) for n in (1 << 10, 1 << 16, 1 << 18, 1 << 20, 1 << 24, 1 << 26)]
        del used
        launch = kda.prepare(*inputs)
        assert launch.plan_counts() == (0, 0, 0) and kda.status_bits(launch) == 0
        assert kda.kernel_error(launch) == 0 and launch.status.tolist() == [0, 0, 0, 0]
        launch()
        torch.cuda.synchronize()
        assert launch.plan_counts()[0] >= len(lens) and kda.status_bits(launch) == 0


@pytest.mark.parametrize("raw", [True, False])
def test_a_call_that_launches_at_once_fills_nothing(kda, raw):
    """The planner writes the status and the counts of every launch before anything reads them, so the one-shot calls enqueue
    the library's kernels and nothing in front of them."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Ops(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.names = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.append(str(func))
            return func(*args, **(kwargs or {}))

    H, lens = 4, [300, 77]
    inputs = to_dev(ko.make_inputs_raw(H, lens, 62))
    plain = plain_on_device(H, sum(lens), 63)
    with Ops() as ops:
        if raw:
            res = kda.run(*inputs)
        else:
            res = kda.chunk_kda(*plain, output_final_state=True, cu_seqlens=inputs[9])
    torch.cuda.synchronize()
    assert res[0].shape == (1, sum(lens), H, 128)
    assert not [n for n in ops.names if any(w in n for w in ("zero", "fill", "copy", "ones", "full"))], ops.names
