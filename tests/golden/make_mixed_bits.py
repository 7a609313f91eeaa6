"""Writes mixed_bits.json: checksums of the mixed form's results, on a GPU.

The file that is committed was written by the engines that the register stages and
the fused radix-3 z pass replaced (shared-memory Stockham, a warp per row, the
unfused z part), so test_gpu_mixed_bits.py holds the new ones to their bits.
Run from the repository's root:  python tests/golden/make_mixed_bits.py
"""
import hashlib
import json
from pathlib import Path

import numpy as np

FILE = Path(__file__).with_name("mixed_bits.json")
GRIDS = [(8, 8, 8), (16, 16, 16), (32, 32, 32), (64, 64, 64), (128, 128, 128), (64, 32, 16),
         (128, 64, 32), (256, 128, 64), (256, 256, 256), (512, 16, 8), (24, 24, 24), (48, 36, 24),
         (96, 64, 48), (72, 72, 72), (96, 96, 96), (144, 96, 72), (192, 128, 96), (288, 24, 24),
         (384, 32, 24), (54, 48, 36), (96, 64, 64), (192, 192, 192), (36, 18, 18)]


def key(n):
    return "x".join(map(str, n))


def checksums(gpu, n):
    """Of the right-hand side (plain, filtered, with output) and of one transform
    each way; inputs are exact FP32 sums of powers of two, the same on every host."""
    ctx = gpu.Context(n=n, precision=gpu.PREC_MIXED)
    rng = np.random.default_rng(sum(n))
    N = ctx.N

    def noise(count):  # uniform in steps of 2^-20
        return rng.integers(-1 << 20, 1 << 20, count) * 2.0 ** -20

    f = np.zeros(ctx.Ntot)
    f[:4 * N] = 2.0 ** -10 * noise(4 * N)
    f[:N] += 1.0
    f[N:2 * N] -= 0.75
    f[4 * N:-1] = 2.0 ** -20 * noise(8 * ctx.M)
    f[-1] = 1.0
    x = noise(N).reshape(n)
    out = []

    def add(a):
        out.append(hashlib.sha256(a.astype(np.float32).tobytes()).hexdigest()[:16])

    for engine in (1, 2) if n[2] == 256 else (0,):
        if engine:
            ctx.set_engine(6, engine)
        for flt, output in ((0, 0), (1, 0), (1, 1)):
            r, ff = ctx.mk_rhs(f, filter=flt, output=output)
            add(r[:-1])
            add(ff[:-1])
        X = ctx.fft(x)
        add(X.view(np.float64))
        add(ctx.ifft(X))
    ctx.close()
    return out


if __name__ == "__main__":
    import sys
    sys.path.insert(0, str(Path.cwd()))
    from instaheat_gb300 import gpu as module
    FILE.write_text(json.dumps({key(n): checksums(module, n) for n in GRIDS}, indent=0) + "\n")
