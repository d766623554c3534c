"""The solves' reciprocal, quotient, square root and exponential equal the
operators and mgcm_rt_exp bit for bit within their ranges: random operands,
special significands, the ends of the ranges, and operands made so that the
exact quotient or root lies as near to the middle of two doubles as it can."""
import ctypes as C
import pathlib
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent
RCP, RCP_SIGNED, QUOT, SQRT, EXP = range(5)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    import torch
    so = tmp_path_factory.mktemp("arith") / "arith_probe.so"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--fmad=false", "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC", "-o", str(so),
                    str(HERE / "arith_probe.cu")], check=True)
    lib = C.CDLL(str(so))
    lib.arith_probe.argtypes = [C.c_int, C.c_longlong] + [C.c_void_p] * 3

    def same(op, b, a=None):
        b = torch.from_numpy(np.ascontiguousarray(b, dtype=np.float64)).cuda()
        a = b if a is None else torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()
        assert a.shape == b.shape and b.numel() > 0
        out = torch.empty((b.numel(), 2), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.arith_probe(op, b.numel(), a.data_ptr(), b.data_ptr(), out.data_ptr()) == 0
        bits = out.view(torch.int64)
        bad = (bits[:, 0] != bits[:, 1]).nonzero().flatten()[:4].cpu().tolist()
        assert not bad, [(float(a[i]).hex(), float(b[i]).hex(), [float(x).hex() for x in out[i]]) for i in bad]
    return same


def _significands(n, rng):
    """Doubles in [1, 2): random ones, those next to 1 and 2, and few-bit ones."""
    near = np.arange(4096, dtype=np.uint64)
    few = np.uint64(1) << rng.integers(0, 52, 4096).astype(np.uint64) | np.uint64(1) << rng.integers(0, 52, 4096).astype(np.uint64)
    frac = np.concatenate([rng.integers(0, 1 << 52, n, dtype=np.uint64), near, np.uint64((1 << 52) - 1) - near, few,
                           np.uint64((1 << 52) - 1) ^ few])
    return (frac | np.uint64(1023 << 52)).view(np.float64)


def _scaled(m, rng, lo, hi):
    """m with exponents over [lo, hi), both ends among them."""
    e = rng.integers(lo, hi, m.size)
    e[:2], e[-2:] = lo, hi - 1
    return np.ldexp(m, e)


def _near_midpoint_quotients(rng):
    """a, b in [1, 2) with a/b = (M + N 2^-54 / B) 2^-54 or 2^-53, M odd, |N| < 16."""
    out = []
    for i in range(3000):
        B = (1 << 52) | int(rng.integers(0, 1 << 52)) | 1
        if i % 2:
            B = (1 << 53) - 1 - 2 * int(rng.integers(0, 1 << (2 + i % 50)))
        for bits in (53, 54):
            inv = pow(B, -1, 1 << bits)
            for N in range(-15, 16, 2):
                M = (-N * inv) % (1 << bits)
                M += (1 << 53) if bits == 53 else 0
                A = (M * B + N) >> bits
                if M >> 53 == 1 and A >> 52 == 1 and (bits == 53 or A < B):
                    assert (A << bits) == M * B + N
                    out.append((A, B))
    return np.ldexp(np.array(out, dtype=np.float64), -52).T


def _near_midpoint_squares():
    """x in [1, 4) whose root is (M + a little) 2^-53, M odd: M^2 = X 2^e - N, |N| < 1024."""
    out = []
    for e in (54, 55):
        for N in range(-1023, 1024):
            if (-N) % 8 != 1:
                continue
            r = 1
            for k in range(3, e):            # Hensel: r^2 = -N modulo 2^e
                if (r * r + N >> k) & 1:
                    r += 1 << (k - 1)
            half = 1 << (e - 1)
            for q in (r % half, -r % half):
                for M in range(q, 1 << 54, half):
                    X = M * M + N >> e
                    if M >> 53 == 1 and X >> 52 == 1 and (M * M + N) % (1 << e) == 0:
                        out.append(np.ldexp(float(X), -52 if e == 54 else -51))
    return np.array(out)


def test_reciprocal(probe):
    rng = np.random.default_rng(1)
    m = _significands(1 << 22, rng)
    probe(RCP, m)
    probe(RCP, _scaled(m, rng, -300, 300))
    probe(RCP_SIGNED, _scaled(m, rng, -300, 300) * rng.choice([-1.0, 1.0], m.size))


def test_quotient(probe):
    rng = np.random.default_rng(2)
    a, b = _near_midpoint_quotients(rng)
    assert a.size > 20000
    probe(QUOT, b, a)
    probe(QUOT, -b, np.ldexp(a, -300))
    b = _significands(1 << 22, rng)
    a = rng.permutation(b)
    probe(QUOT, b, a)
    probe(QUOT, _scaled(b, rng, -300, 300), _scaled(a, rng, -300, 300) * rng.choice([-1.0, 1.0], a.size))
    probe(QUOT, b, np.zeros_like(b))


def test_square_root(probe):
    rng = np.random.default_rng(3)
    x = _near_midpoint_squares()
    assert x.size > 300
    for e in (-300, -2, 0, 296):
        probe(SQRT, np.ldexp(x, e))
    m = _significands(1 << 22, rng)
    probe(SQRT, _scaled(m, rng, -300, 300))
    r = _significands(1 << 20, rng)
    probe(SQRT, r * r)


def test_exponential(probe):
    rng = np.random.default_rng(4)
    step = np.log(2.0) / 32
    k = np.arange(-32318, 32318) * step          # the edges of the table's intervals lie between these
    x = np.concatenate([rng.uniform(-700.0, 700.0, 1 << 22), rng.uniform(-36.0, 36.0, 1 << 22), k, k + step / 2,
                        np.nextafter(k + step / 2, 1e9), np.nextafter(k + step / 2, -1e9),
                        rng.choice([-1.0, 1.0], 4096) * np.ldexp(rng.uniform(1, 2, 4096), rng.integers(-1022, 9, 4096)),
                        [0.0, -0.0, 5e-324, -5e-324, np.nextafter(700.0, 0.0), -np.nextafter(700.0, 0.0)]])
    probe(EXP, x[np.abs(x) < 700.0])
