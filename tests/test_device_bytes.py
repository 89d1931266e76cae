"""spns_estimate_device_bytes counts what a box allocates at creation (no GPU needed)."""
import math
import os

import pytest

from gpu_util import make_args
from spns_b200 import hit


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("N", [(32, 32, 32), (64, 96, 128), (32, 32, 512)])
def test_estimate_counts_arrays_and_twiddle_tables(N, precision):
    if not os.path.exists(hit.LIB_PATH):
        pytest.skip("libspns.so not built")
    args = make_args(0, Ns=N, les=0.17)                    # (no aliasing planes)
    M = (args.Mx, args.My, args.Mz)
    cs = 16 if precision == 0 else 8                       # bytes of a complex value
    Kx, Ky, Kz = N[0] // 2 * 2 + 1, N[1] // 2 * 2 + 1, N[2] // 2 + 1
    unit = (128 if Kz * cs >= 1024 else 32) // cs          # rows of the work buffers are padded to whole units
    Kp = -(-Kz // unit) * unit
    arrays = cs * 3 * Ky * Kx * Kz * (2 if precision == 0 else 3)        # u [and its low part], R
    arrays += cs * (6 * Ky * M[0] * Kp + 9 * M[1] * M[0] * Kp)
    arrays += 16 * (math.ceil(math.sqrt(sum((n // 2) ** 2 for n in N))) + 1)   # E(K), Om(K) of the shells
    # a table per length: every divisor above 1 for the powers 1, 2, 4 and 8; in single precision once more as pairs
    entries = sum(4 * sum(d for d in range(2, L + 1) if L % d == 0) for L in set(M))
    tables = cs * entries * (1 if precision == 0 else 3)
    est = hit.estimate_device_bytes(args, precision=precision)
    assert arrays + tables <= est <= arrays + tables + 4096              # (the solver scalars)

