"""Sums of more operands than one launch's parameters hold: their sources go to
the device in one copy, whatever blocks the operands hold.  Operands that hold
different blocks (a run a block) then cost two or three launches more than
operands that hold the same (one run), not a copy and a wait for each block:
within three times the latter's time, with the operands marshalled beforehand.
The result is that of the same sum in parts of few operands to rounding: two
orders of n terms differ by at most 2 n 2^-53 sum |coef x|."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [161, 200])
def test_many_operands_one_copy(su2lib, n):
    import torch

    from su2dmrg_gb300 import capi
    from su2dmrg_gb300 import su2 as S

    rng = np.random.default_rng(n)
    b = lambda d: S.Su2Bond(d, list(range(13)), [5] * 13)
    struct = lambda: S.Su2Struct([b(1), S.Su2Bond(1, [2], [1]), b(-1)], 0).with_legal_flags()
    coefs = rng.standard_normal(n)

    def timed(mixed):
        ops = []
        for i in range(n):
            s = struct()
            legal = np.flatnonzero(s.flag)
            if mixed:
                s.flag = (s.flag * (rng.random(len(s.flag)) < 0.6)).astype(np.int32)
                s.flag[legal[i % len(legal)]] = 1
            ops.append((s, torch.randn(s.size(), dtype=torch.float64, device="cuda")))
        keep = []
        arr = (capi.Tensor * n)(*[S._tensor(s, x, keep) for s, x in ops])
        c = (ctypes.c_double * n)(*coefs)
        out = torch.full((struct().size(),), float("nan"), dtype=torch.float64, device="cuda")
        f = capi.lib().su2g_operator_combine
        call = lambda: capi.check(f(n, ctypes.addressof(arr), ctypes.addressof(c), out.data_ptr(),
                                    torch.cuda.current_stream().cuda_stream))
        took = []
        for _ in range(30):
            torch.cuda.synchronize()
            t = time.perf_counter()
            call()
            took.append(time.perf_counter() - t)
        parts = torch.zeros_like(out)
        size = torch.zeros_like(out)
        off, _ = struct().offsets()
        for (s, x), ci in zip(ops, coefs):
            o, _ = s.offsets()
            for k in np.flatnonzero(s.flag):
                m = int(np.prod(s.block_shape(int(k))))
                parts[int(off[k]): int(off[k]) + m] += ci * x[int(o[k]): int(o[k]) + m]
                size[int(off[k]): int(off[k]) + m] += (ci * x[int(o[k]): int(o[k]) + m]).abs()
        assert bool(((out - parts).abs() <= 2 * n * 2.0**-53 * size).all())
        return float(np.median(took))

    equal, mixed = timed(False), timed(True)
    print(f"n = {n}: equal {equal * 1e6:.1f} us, mixed {mixed * 1e6:.1f} us")
    assert mixed <= 3 * equal
