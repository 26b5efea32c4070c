"""The LIBSVM parser's windows at their edges: tokens per line and per 512-byte window around multiples of 32 (a window's
tokens past the last 32 are left to the next one), tokens of every length across the boundaries, values of 8 to 20
significant digits before and after the point, indices of up to 12 digits' width, repeated and decreasing indices.
Bit for bit against the reader oracle."""
import numpy as np
import pytest

from test_libsvm_gpu import gpu_parse, oracle_read, same_bits

pytestmark = pytest.mark.gpu


def _text(seed, counts, blanks, order):
    g = np.random.default_rng(seed)
    rows = []
    for k in counts:
        idx = np.arange(1, k + 1)
        if order == "shuffled":
            idx = g.integers(1, 201, k)
        row = ["+1" if g.random() < 0.5 else "-1"]
        for i in idx:
            digits = "".join(g.choice(list("0123456789"), g.integers(1, 21)))
            at = int(g.integers(0, len(digits) + 1))
            value = digits[:at] + ("." if g.random() < 0.8 else "") + digits[at:]
            row.append("0" * int(g.integers(0, 10) if g.random() < 0.1 else 0) + f"{i}:{value}")
        rows.append((" " * blanks).join(row) + " " * int(g.integers(0, 2)))
    return ("\n".join(rows) + "\n").encode()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("blanks,order,offset", [(1, "rising", 0), (3, "rising", 5), (1, "shuffled", 0)])
def test_windows(gpu_ctx, dt, blanks, order, offset):
    counts = [0, 1, 30, 31, 32, 33, 63, 64, 65, 95, 96, 127, 128, 129, 200, 160]
    text = _text(3 + blanks, counts * 3, blanks, order)
    n, d = 3 * len(counts), 200
    Xo, Yo, lo = oracle_read(text, n, d, dt)
    Xg, Yg, lg = gpu_parse(gpu_ctx, text, n, d, dt, offset)
    assert lg == lo
    assert same_bits(Xg, Xo, dt) and same_bits(Yg, Yo, dt)


def test_dense_short_tokens(gpu_ctx):
    # four-byte tokens: 128 and more of them start in one window
    text = b"".join(b"1 " + b" ".join(b"%d:%d" % (i + 1, i % 10) for i in range(9)) * 1 + b"\n" for _ in range(40))
    text += b"1 " + b" ".join(b"%d:%d" % (i % 9 + 1, i % 10) for i in range(700)) + b"\n"
    Xo, Yo, lo = oracle_read(text, 41, 9, np.float32)
    Xg, Yg, lg = gpu_parse(gpu_ctx, text, 41, 9, np.float32)
    assert lg == lo and same_bits(Xg, Xo, np.float32) and same_bits(Yg, Yo, np.float32)
