"""Sizes of the optional scratch, on the host alone."""
import pytest


@pytest.mark.parametrize("op,bytes_per_pixel", [(1, 128), (2, 160), (3, 64)])
def test_no_staging_beyond_32_bit_row_offsets(op, bytes_per_pixel):
    """Pooling, argmax backward, scatter: scratch is reported for groups of planes below 4 GiB, which the entry points use, and
    not for larger ones, which they do not."""
    from sphmap import capi
    n = (1 << 32) // bytes_per_pixel
    bytes_for = lambda pixels: capi.lib.sph_staging_bytes(capi._int(op), *capi._ints(32, pixels, 9 * pixels), capi._int(capi.F32))  # noqa: E731
    assert (1 << 32) > bytes_for(n - 8) >= (n - 8) * bytes_per_pixel
    assert bytes_for(n) == 0 and bytes_for(2 * n) == 0
