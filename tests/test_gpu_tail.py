"""Whole float chains against the oracle where the tail, the box kernel and the returned levels can go wrong: chains
that are all tail, one-texel-wide ones, windows too many for the tail's table, odd box sizes from the input's
bytes, and an output off its 16-byte boundary."""
import numpy as np
import pytest

import ntg
import ntg.synth as synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZES = [(64, 64), (1, 1024), (2048, 1), (33, 31), (7, 500), (96, 40), (3, 2), (130, 127)]
FILTERS = [(ntg.FILTER_BOX, 0.5), (ntg.FILTER_TRIANGLE, 1.0), (ntg.FILTER_KAISER, 3.0), (ntg.FILTER_KAISER, 6.0)]


def ntg_steps(n):
    """The extents that a chain halves."""
    out = []
    while n > 1:
        out.append(n)
        n //= 2
    return out


@pytest.mark.parametrize("filt,width", FILTERS)
@pytest.mark.parametrize("wrap", [0, 1, 2])
def test_chain_levels_match_oracle(ctx, oracle, filt, width, wrap):
    for i, (w, h) in enumerate(SIZES):
        img = synth.colour_texture(w, h, 10 * i + wrap, alpha=np.random.default_rng(i).integers(0, 256, (h, w)).astype(np.uint8))
        xform = i % 3
        opt = ntg.ChainOptions.make(format=ntg.FORMAT_BC1, filter=filt, filter_width=width, params=(4.0, 1.0), wrap=wrap,
                                    in_xform=xform, out_xform=xform)
        levels, _ = oracle.mip_chain(img, w, h, filt, width, 4.0, 1.0, wrap, 0, xform, xform)
        ref = np.concatenate([lv.reshape(-1) for lv in levels])
        buf = torch.zeros(ref.size + 2, dtype=torch.float32, device="cuda")
        if width == 6.0 and any(n > 1 and 12.0 * n / (n // 2) + 2 > 32 for n in ntg_steps(w) + ntg_steps(h)):
            with pytest.raises(ntg.NtgError) as e:  # windows wider than 32 taps are refused
                ctx.mip_chain(torch.from_numpy(img).cuda(), w, h, opt, out=buf[:ref.size])
            assert e.value.code == ntg.NTG_ERROR_UNSUPPORTED_FEATURE
            continue
        for offset in (0, 1):
            out = ctx.mip_chain(torch.from_numpy(img).cuda(), w, h, opt, out=buf[offset:offset + ref.size])
            assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32)), (w, h, offset)
