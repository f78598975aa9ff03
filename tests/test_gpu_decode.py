"""Decoding and error sums at the edges of their 16-byte paths: widths of whole fours with ragged heights,
odd widths, planes off their 16-byte boundary, infinities and sums beyond float's range."""
import numpy as np
import pytest

import ntg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("fmt", [1, 2, 4, 6, 7])
@pytest.mark.parametrize("w,h,offset", [(64, 30, 0), (64, 30, 1), (4, 1, 0), (45, 27, 0), (132, 7, 2)])
def test_decode_matches_oracle(ctx, oracle, fmt, w, h, offset):
    rng = np.random.default_rng(fmt * 100 + w)
    blocks = rng.integers(0, 256, ntg.BLOCK_BYTES[fmt] * ntg.nblocks(w, h)).astype(np.uint8)
    buf = torch.zeros(4 * w * h + 4, dtype=torch.float32, device="cuda")
    out = buf[offset:offset + 4 * w * h]
    ctx.decode(fmt, torch.from_numpy(blocks).cuda(), w, h, out=out)
    ref = oracle.decode(fmt, blocks, w, h)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), np.asarray(ref).reshape(-1).view(np.uint32))
    assert not buf[4 * w * h + offset:].any() and not buf[:offset].any()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("w,h,offset", [(64, 32, 0), (64, 32, 1), (45, 27, 0), (1, 1, 0), (1024, 700, 0)])
def test_error_sums_match_float64(ctx, w, h, offset, mode):
    rng = np.random.default_rng(w + h)
    n = w * h
    a, b = (rng.random(4 * n).astype(np.float32) for _ in range(2))

    def sums(a, b):
        da, db = (torch.zeros(4 * n + 4, dtype=torch.float32, device="cuda") for _ in range(2))
        da[offset:offset + 4 * n] = torch.from_numpy(a)
        db[offset:offset + 4 * n] = torch.from_numpy(b)
        return ctx.error_sums(da[offset:offset + 4 * n], db[offset:offset + 4 * n], w, h, alpha_mode=mode).cpu().numpy()

    def ref(a, b):  # every term rounded to float as the kernel rounds it, the sum in 64 bits
        a, b = a.reshape(4, n), b.reshape(4, n)
        wgt = a[3] * a[3] if mode else np.ones(n, np.float32)
        with np.errstate(over="ignore", invalid="ignore"):
            d = a[:3] - b[:3]
            return (((d * d) * wgt).astype(np.float64).sum(), (((b[3] - a[3]) ** 2).astype(np.float64)).sum())

    # 64-bit sums of at most 2.2 million terms, in any order: 2^-53 x 2^21 relative
    np.testing.assert_allclose(sums(a, b), ref(a, b), rtol=2.4e-10)
    a[0] = np.float32(1.8e19)  # squares near float's largest: a few of them pass it
    a[n // 2] = np.float32(1.8e19)
    a[n] = np.float32(1.8e19)
    np.testing.assert_allclose(sums(a, b), ref(a, b), rtol=2.4e-10)
    a[0] = np.inf
    got, want = sums(a, b), ref(a, b)
    assert got[0] == want[0] == np.inf and np.isclose(got[1], want[1], rtol=2.4e-10)


def test_error_sums_lose_no_bits_of_double(ctx):
    """One step of the kernel, squares of unlike size: the sums of a thread's 12 and 4 terms are as exact as double
    additions make them, 2^-53 for each; and of a whole image, whose longest chain of additions in double would be the
    112 terms of a thread and the 26 of its CTA and the atomics'."""
    import math
    for w, h, seeds, steps in [(2, 2, 64, 12), (1024, 1024, 2, 200)]:
        n = w * h
        for seed in range(seeds):
            rng = np.random.default_rng(seed)
            a = (rng.random(4 * n) * 10.0 ** -rng.uniform(0, 4, 4 * n)).astype(np.float32)
            d = torch.from_numpy(a).cuda()
            got = ctx.error_sums(d, torch.zeros_like(d), w, h).cpu().numpy()
            terms = (a * a).reshape(4, n)
            for have, want in zip(got, (math.fsum(map(float, terms[:3].reshape(-1))), math.fsum(map(float, terms[3])))):
                assert abs(have - want) <= steps * 2.0 ** -53 * want, (w, seed)
