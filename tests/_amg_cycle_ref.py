"""Test infrastructure: a numpy restatement of the V-cycle as the solvers apply
it (chuanflow_b200/csrc/amg.cu), on the hierarchy of _amg_ref: several weighted
sweeps before and after the correction on the coarse levels, Chebyshev weights
over [lo, 1.9], chosen by the operator's skew class and the size of the first
coarse level.  In FP32 like the device, or with the same FP32 operators in
FP64, which gives the rounding error of either."""
import numpy as np

import _amg_ref as R

SELL_MIN_ROWS = 32768
FOUR_MIN_ROWS = 100000


def chebyshev(m, lo, hi=1.9):
    return [1.0 / (0.5 * (hi + lo) + 0.5 * (hi - lo) * np.cos(np.pi * (2 * k + 1) / (2 * m))) for k in range(m)]


def weights(rows, skew_class):
    """Per aggregated level (the finest first): its sweeps' weights."""
    if skew_class == 2 or (skew_class == 1 and rows[1] < SELL_MIN_ROWS):
        first = rest = [0.8]
    else:
        lo2, lo4 = (0.3, 0.3) if skew_class == 1 else (0.2, 0.1)
        rest = chebyshev(2, lo2)
        first = rest if rows[1] < SELL_MIN_ROWS else chebyshev(4 if skew_class == 1 or rows[1] >= FOUR_MIN_ROWS else 3, lo4)
    return [[0.8]] + [first] + [rest] * len(rows)


class Cycle:
    def __init__(self, H, skew_class, dtype):
        self.w = weights(H.rows, skew_class)
        self.t = dtype
        self.levels = [{"A": lv["A"].astype(dtype), "dinv": lv["dinv"].astype(dtype), "P": lv["P"].astype(dtype)}
                       for lv in H.levels]
        self.dense = H.dense.astype(dtype)

    def __call__(self, r, level=0):
        b = r.astype(np.float32).astype(self.t) if level == 0 else r
        if level == len(self.levels):
            return self.dense @ b
        A, dinv, P = (self.levels[level][k] for k in ("A", "dinv", "P"))
        w = [self.t(np.float32(v)) for v in self.w[level]]
        x = w[0] * dinv * b
        for v in w[1:]:
            x = x + v * dinv * (b - A @ x)
        y = x + self.t(R.SCALE) * (P @ self(P.T @ (b - A @ x), level + 1))
        for v in w[::-1]:
            y = y + v * dinv * (b - A @ y)
        return y
