"""Sums of block tensors whose operands hold different blocks: one run of equal
flags, runs that break at every block, more runs and more sources than one
launch's parameters hold (32 and 160), one-element blocks and tile edges, and
the output written over an operand.

Every element is one chain of fused multiply-adds in operand order, so
the result lies within n * 2^-53 * sum |coef x| of the exact sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _struct(S, dims):
    b = lambda d: S.Su2Bond(d, list(range(len(dims))), list(dims))
    return S.Su2Struct([b(1), S.Su2Bond(1, [2], [1]), b(-1)], 0).with_legal_flags()


@pytest.mark.parametrize("dims", [[1, 1], [1, 2, 3], [16, 32, 17], [3, 511, 1], [5] * 23])
@pytest.mark.parametrize("n", [1, 2, 7, 160, 161, 325])
@pytest.mark.parametrize("flags", ["equal", "mixed"])
def test_sum_of_runs(su2lib, dims, n, flags):
    import torch

    from su2dmrg_gb300 import su2 as S

    rng = np.random.default_rng(len(dims) * 1000 + n)
    ref = _struct(S, dims)
    legal = np.flatnonzero(ref.flag)
    ops, dense, coefs = [], [], rng.standard_normal(n)
    off, total = ref.offsets()
    size = {b: int(np.prod(ref.block_shape(b))) for b in legal}
    for i in range(n):
        s = _struct(S, dims)
        if flags == "mixed":
            s.flag = s.flag * (rng.random(len(s.flag)) < 0.6)
            s.flag[legal[i % len(legal)]] = 1
            s.flag = s.flag.astype(np.int32)
        o, t = s.offsets()
        x = rng.standard_normal(t)
        full = np.zeros(total)
        for b in legal:
            if s.flag[b]:
                full[off[b]:off[b] + size[b]] = x[o[b]:o[b] + size[b]]
        ops.append((s, torch.from_numpy(x).cuda()))
        dense.append(full)
    st, y = S.operator_combine(ops, coefs)
    want = np.zeros(total, np.longdouble)
    mag = np.zeros(total)
    for c, d in zip(coefs, dense):
        want += np.longdouble(c) * d
        mag += np.abs(c * d)
    o, t = st.offsets()
    got = y.cpu().numpy()[:t]
    for b in legal:
        if st.flag[b]:
            a = slice(off[b], off[b] + size[b])
            err = np.abs(got[o[b]:o[b] + size[b]] - want[a])
            assert (err <= (n + 1) * 2.0 ** -53 * mag[a]).all(), b
        else:
            assert not any(s.flag[b] for s, _ in ops)
