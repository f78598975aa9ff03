"""The cluster fits' scan (ntg_scan.cuh) against the oracle, block for block, on the contents whose bounds
are tightest: nearly flat blocks (every ordering a possible winner), end points on snapping ties, tiny and
unequal weights, colours below the black threshold, values outside [0, 1], NaN and infinities; and on block
counts that leave a warp's second half or a CTA's last warps without a block."""
import numpy as np
import pytest

import ntg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def contents(kind, w, h, seed):
    rng = np.random.default_rng(seed)
    rgb = rng.random((3, h, w)).astype(np.float32)
    a = rng.random((h, w)).astype(np.float32)
    if kind == "flat":        # a few steps of 1 / 255 around a colour
        rgb = (0.5 + rng.integers(-1, 2, (3, h, w)) / 255.0).astype(np.float32)
    elif kind == "faint":     # just above the merging threshold
        rgb = (rng.random((3, 1, 1)) + rng.random((3, h, w)) / 60.0).astype(np.float32)
    elif kind == "grid":      # colours on the 5:6:5 grid and half way between its points
        rgb = np.stack([rng.integers(0, 63, (h, w)) / 62.0, rng.integers(0, 127, (h, w)) / 126.0,
                        rng.integers(0, 63, (h, w)) / 62.0]).astype(np.float32)
    elif kind == "dark":
        rgb *= 0.2
    elif kind == "weights":   # alphas over five orders of magnitude
        a = (10.0 ** -rng.uniform(0, 5, (h, w))).astype(np.float32)
    elif kind == "wide":      # beyond what the scan's bound covers
        rgb = (rgb * 6 - 3).astype(np.float32)
    elif kind == "odd":
        rgb[rng.random(rgb.shape) < 0.05] = np.nan
        rgb[rng.random(rgb.shape) < 0.02] = np.inf
    elif kind == "ramp":      # noise around a gradient, as smooth textures have it
        rgb = (0.3 + 0.4 * (np.arange(w)[None, None, :] / w) + rng.uniform(-8, 8, (3, h, w)) / 255.0).astype(np.float32)
    if kind != "weights":
        a[rng.random((h, w)) < 0.1] = 0
    return np.concatenate([rgb.reshape(-1), a.reshape(-1)]).astype(np.float32)


KINDS = ["noise", "flat", "faint", "grid", "dark", "weights", "wide", "odd", "ramp"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("fmt", [ntg.FORMAT_BC1, ntg.FORMAT_BC1A, ntg.FORMAT_BC3])
def test_fits_match_oracle(ctx, oracle, kind, fmt):
    image = {ntg.FORMAT_BC1: oracle.bc1_image, ntg.FORMAT_BC3: oracle.bc3_image,
             ntg.FORMAT_BC1A: lambda i, w, h, alpha, q, **kw: oracle.bc1a_image(i, w, h, alpha, **kw)}[fmt]
    for i, (w, h) in enumerate([(4, 4), (8, 4), (12, 4), (28, 4), (36, 4), (61, 35), (128, 96)]):
        img = contents(kind, w, h, 100 * i + len(kind))
        for quality, alpha, cw in [(1, 0, (1, 1, 1)), (1, 1, (1, 1, 1)), (2, 1, (0.6, 1.0, 0.4))]:
            if quality == 2 and w > 61:
                continue
            got = ctx.encode(fmt, torch.from_numpy(img).cuda(), w, h, quality=quality, alpha_mode=alpha, cw=cw)
            ref = image(img, w, h, alpha, quality, cw=cw, threads=8)
            assert np.array_equal(got.cpu().numpy(), ref), (kind, w, h, quality, alpha)


def test_bc1a_every_split_a_candidate(ctx, oracle):
    """Nearly flat blocks with unequal weights: every split of both fits, and the repeats that fill the tables' last rows,
    are possible winners, as many as the list of them can hold."""
    w, h = 4, 4 * 6083
    img = contents("faint", w, h, 6088)
    got = ctx.encode(ntg.FORMAT_BC1A, torch.from_numpy(img).cuda(), w, h, quality=1, alpha_mode=1)
    assert np.array_equal(got.cpu().numpy(), oracle.bc1a_image(img, w, h, 1, threads=8))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("fmt", [ntg.FORMAT_BC1A, ntg.FORMAT_BC3])
def test_squish_launch_sizes_agree(ctx, fmt, kind):
    """The two kernels of the squish fits, which share the work by launch size (68,096 blocks), over the same blocks;
    among them ("weights") single points of so tiny a weight that their axis is NaN."""
    w, h = 4, 4 * 60000
    img = torch.from_numpy(contents(kind, w, h, 3007)).cuda().reshape(4, h, w)
    small = ctx.encode(fmt, img, w, h, quality=1, alpha_mode=1)
    img = torch.cat([img, img[:, :4 * 8097]], 1).contiguous()
    large = ctx.encode(fmt, img, w, 4 * 68097, quality=1, alpha_mode=1)
    assert torch.equal(large[:small.numel()], small)


@pytest.mark.parametrize("blocks", [3040, 3041, 6083])
@pytest.mark.parametrize("fmt", [ntg.FORMAT_BC1, ntg.FORMAT_BC1A, ntg.FORMAT_BC3])
def test_blocks_per_warp(ctx, oracle, fmt, blocks):
    """Where launches go from one block per warp to two (3,040 blocks), and an odd count above it."""
    image = {ntg.FORMAT_BC1: oracle.bc1_image, ntg.FORMAT_BC3: oracle.bc3_image,
             ntg.FORMAT_BC1A: lambda i, w, h, alpha, q, **kw: oracle.bc1a_image(i, w, h, alpha, **kw)}[fmt]
    w, h = 4, 4 * blocks
    for kind in KINDS:
        img = contents(kind, w, h, blocks + len(kind))
        got = ctx.encode(fmt, torch.from_numpy(img).cuda(), w, h, quality=1, alpha_mode=1)
        assert np.array_equal(got.cpu().numpy(), image(img, w, h, 1, 1, threads=8)), kind


@pytest.mark.parametrize("kind", KINDS)
def test_bc1_one_block_per_thread(ctx, oracle, kind):
    """BC1 launches of 150,000 blocks and more, an odd count of them, against the oracle."""
    w, h = 4, 4 * 150001
    img = contents(kind, w, h, 77)
    for alpha, cw in [(1, (1, 1, 1)), (0, (0.6, 1.0, 0.4))]:
        got = ctx.encode(ntg.FORMAT_BC1, torch.from_numpy(img).cuda(), w, h, quality=1, alpha_mode=alpha, cw=cw)
        assert np.array_equal(got.cpu().numpy(), oracle.bc1_image(img, w, h, alpha, 1, cw=cw, threads=16)), alpha


@pytest.mark.parametrize("xform", [ntg.XFORM_NONE, ntg.XFORM_SRGB])
@pytest.mark.parametrize("size", [8, 200, 700, 1700])
def test_listed_blocks_get_the_full_fit(ctx, size, xform):
    """The learned path's fallbacks: with a margin that lists every block the result is the plain fit's, at 1700x1700 from lists
    of more than 150,000 blocks (240,833), which a kernel of their own takes, or with a transform more blocks than the grid."""
    rng = np.random.default_rng(size)
    img = torch.from_numpy(rng.integers(0, 256, (size, size, 4), dtype=np.uint8)).cuda()
    opt = ntg.ChainOptions.make(format=ntg.FORMAT_BC1, in_xform=xform, out_xform=xform)
    net = ntg.MLP(seed=1)
    try:
        got, stats = ctx.compress_chain_learned(net, img, size, size, opt, radius=1, margin=-1.0)
        assert size == 8 or stats["full_fit"] > 9 * stats["kept"]  # a block that its palette holds exactly is not listed
        assert torch.equal(got, ctx.compress_chain(img, size, size, opt))
    finally:
        net.close()


@pytest.mark.parametrize("cw", [(3, 3, 3), (0.1, 5, 2), (100, 1, 0), (2e5, 1e6, 9e5), (1e7, 1e7, 1e7)])
@pytest.mark.parametrize("fmt", [ntg.FORMAT_BC1, ntg.FORMAT_BC1A, ntg.FORMAT_BC3])
def test_colour_weights_of_any_size(ctx, oracle, fmt, cw):
    """Colour weights above 1, whose squares scale the scan's errors and bound: up to the largest that it takes (2^20)
    and beyond it."""
    image = {ntg.FORMAT_BC1: oracle.bc1_image, ntg.FORMAT_BC3: oracle.bc3_image,
             ntg.FORMAT_BC1A: lambda i, w, h, alpha, q, **kw: oracle.bc1a_image(i, w, h, alpha, **kw)}[fmt]
    w, h = 61, 130
    for kind in KINDS:
        img = contents(kind, w, h, len(kind))
        for alpha in (0, 1):
            got = ctx.encode(fmt, torch.from_numpy(img).cuda(), w, h, quality=1, alpha_mode=alpha, cw=cw)
            assert np.array_equal(got.cpu().numpy(), image(img, w, h, alpha, 1, cw=cw, threads=8)), (kind, alpha)
