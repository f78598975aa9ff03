"""Chains whose first levels are encoded beside the filters of the others, against the same calls with the phases timed,
which run one after the other: at the sizes where the rule changes, odd extents, chains without a tail, and calls from
several threads and streams on one context."""
import threading

import numpy as np
import pytest

import ntg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def image(w, h, seed):
    rng = np.random.default_rng(seed)
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[: h // 2] = img[: h // 2] // 16 + 100  # half of it nearly flat
    return torch.from_numpy(img).cuda()


def serial(ctx, img, w, h, opt):
    ctx.profile(True)
    try:
        return ctx.compress_chain(img, w, h, opt)
    finally:
        ctx.profile(False)


SIZES = [(1, 1), (2, 5), (4, 4), (16, 16), (33, 64), (65, 65), (64, 1), (200, 120), (444, 440), (448, 439), (512, 512),
         (513, 770), (1366, 769), (1500, 3)]


@pytest.mark.parametrize("fmt", [ntg.FORMAT_BC1, ntg.FORMAT_BC1A, ntg.FORMAT_BC3, ntg.FORMAT_BC4, ntg.FORMAT_BC5])
@pytest.mark.parametrize("filt", [ntg.FILTER_BOX, ntg.FILTER_KAISER])
def test_chain(ctx, fmt, filt):
    for i, (w, h) in enumerate(SIZES):
        img = image(w, h, i)
        for quality, x, levels in [(1, ntg.XFORM_SRGB, 0), (0, ntg.XFORM_NONE, 0), (1, ntg.XFORM_GAMMA, 2), (1, ntg.XFORM_NONE, 1)]:
            if fmt == ntg.FORMAT_BC1A and quality == 0:
                continue
            opt = ntg.ChainOptions.make(format=fmt, quality=quality, filter=filt, alpha_mode=ntg.ALPHA_TRANSPARENCY, in_xform=x,
                                        out_xform=x, max_levels=levels)
            assert torch.equal(ctx.compress_chain(img, w, h, opt), serial(ctx, img, w, h, opt)), (w, h, quality, levels)


@pytest.mark.parametrize("fmt,size", [(ntg.FORMAT_BC5, 1452), (ntg.FORMAT_BC3, 912), (ntg.FORMAT_BC3, 916), (ntg.FORMAT_BC1, 2048)])
def test_large(ctx, fmt, size):
    img = image(size, size, 9)
    opt = ntg.ChainOptions.make(format=fmt, filter=ntg.FILTER_TRIANGLE)
    assert torch.equal(ctx.compress_chain(img, size, size, opt), serial(ctx, img, size, size, opt))


def test_streams_and_threads(ctx):
    """Each thread's chains on its own stream and context, and the results read on that stream straight away."""
    errors = []

    def work(k):
        own = ntg.Context(0)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for i in range(6):
                w, h = [(64, 64), (512, 512), (700, 300)][(i + k) % 3]
                opt = ntg.ChainOptions.make(format=[ntg.FORMAT_BC1, ntg.FORMAT_BC3][k % 2])
                img = image(w, h, 10 * k + i)
                got = own.compress_chain(img, w, h, opt).clone()
                img.zero_()  # ordered after the call
                stream.synchronize()
                if not torch.equal(got, serial(own, image(w, h, 10 * k + i), w, h, opt)):
                    errors.append((k, i))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


@pytest.mark.parametrize("filt", [ntg.FILTER_BOX, ntg.FILTER_KAISER])
def test_levels(ctx, filt):
    """Returned levels: level 0 is written beside the filters of the others."""
    for w, h in [(1, 1), (2, 5), (65, 65), (513, 770), (1024, 1024)]:
        img = image(w, h, w)
        for levels in (0, 1, 2):
            opt = ntg.ChainOptions.make(filter=filt, in_xform=ntg.XFORM_SRGB, max_levels=levels)
            got = ctx.mip_chain(img, w, h, opt)
            ctx.profile(True)
            try:
                assert torch.equal(got, ctx.mip_chain(img, w, h, opt)), (w, h, levels)
            finally:
                ctx.profile(False)


@pytest.mark.parametrize("filt", [ntg.FILTER_BOX, ntg.FILTER_TRIANGLE, ntg.FILTER_KAISER])
def test_levels_sharing_sectors(ctx, filt):
    """Returned levels whose boundaries fall inside a 32-byte sector (an odd number of texels so far), two images in turn
    into one buffer, so that a sector read before its level is written still holds the other image's."""
    for w, h in [(513, 513), (1025, 771), (257, 1027)]:
        opt = ntg.ChainOptions.make(filter=filt)
        images = [image(w, h, 2 * w), image(w, h, 2 * w + 1)]
        ctx.profile(True)
        try:
            want = [ctx.mip_chain(i, w, h, opt).clone() for i in images]
        finally:
            ctx.profile(False)
        out = torch.zeros_like(want[0])
        for k in range(20):
            assert torch.equal(ctx.mip_chain(images[k & 1], w, h, opt, out=out), want[k & 1]), (w, h, k)


def test_streams_on_one_context(ctx):
    """Calls on several streams of one context, no synchronisation between them: each waits for the one before, whose
    workspace and job lists it would overwrite. Small and large calls in turn, so that the workspace and the lists grow (and
    are freed) under a running call too."""
    calls = []
    for k, (w, h, fmt) in enumerate([(1024, 1024, ntg.FORMAT_BC3), (64, 64, ntg.FORMAT_BC1), (1500, 700, ntg.FORMAT_BC1),
                                     (256, 256, ntg.FORMAT_BC5), (2048, 1024, ntg.FORMAT_BC1), (333, 517, ntg.FORMAT_BC3)]):
        opt = ntg.ChainOptions.make(format=fmt, filter=ntg.FILTER_KAISER, in_xform=ntg.XFORM_SRGB, out_xform=ntg.XFORM_SRGB)
        calls.append((image(w, h, k), w, h, opt))
    want = [serial(ctx, *c) for c in calls]
    own = ntg.Context(0)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got = []
    for k in range(4 * len(calls)):
        with torch.cuda.stream(streams[k % 3]):
            got.append(own.compress_chain(*calls[k % len(calls)]))
    torch.cuda.synchronize()
    for k, blocks in enumerate(got):
        assert torch.equal(blocks, want[k % len(calls)]), k

    errors = []

    def work(t):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for k in range(8):
                blocks = own.compress_chain(*calls[(k + t) % len(calls)])
                stream.synchronize()
                if not torch.equal(blocks, want[(k + t) % len(calls)]):
                    errors.append((t, k))
    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    own.close()


@pytest.mark.parametrize("filt", [ntg.FILTER_BOX, ntg.FILTER_KAISER])
@pytest.mark.parametrize("where", [0, 1])
def test_levels_over_the_image(ctx, filt, where):
    """Levels returned into the buffer that holds the image, at its start or its end."""
    for w, h in [(64, 64), (65, 33), (512, 300), (1024, 1024)]:
        img = image(w, h, w + h)
        opt = ntg.ChainOptions.make(filter=filt)
        want = ctx.mip_chain(img, w, h, opt)
        buf = torch.empty_like(want)
        at = 0 if where == 0 else buf.numel() - w * h
        inside = buf[at:at + w * h]
        inside.copy_(img.reshape(-1).view(torch.float32))
        assert torch.equal(ctx.mip_chain(inside, w, h, opt, out=buf), want), (w, h)


@pytest.mark.parametrize("fmt", [ntg.FORMAT_BC1, ntg.FORMAT_BC1A, ntg.FORMAT_BC3, ntg.FORMAT_BC4, ntg.FORMAT_BC5])
@pytest.mark.parametrize("filt", [ntg.FILTER_BOX, ntg.FILTER_KAISER])
def test_small(ctx, fmt, filt):
    """Both sides of the smallest overlapped chains, 200 and 400 blocks."""
    for i, (w, h) in enumerate([(56, 55), (57, 53), (79, 80), (81, 76), (97, 66), (800, 4), (3, 801)]):
        img = image(w, h, i)
        for x, levels in [(ntg.XFORM_SRGB, 0), (ntg.XFORM_NONE, 3)]:
            opt = ntg.ChainOptions.make(format=fmt, filter=filt, alpha_mode=ntg.ALPHA_TRANSPARENCY, in_xform=x, out_xform=x,
                                        max_levels=levels)
            assert torch.equal(ctx.compress_chain(img, w, h, opt), serial(ctx, img, w, h, opt)), (w, h, levels)
