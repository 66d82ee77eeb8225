"""Which form a tensor-parallel product takes whose ranks are all in one launch on one GPU."""


def test_long_sums_of_few_tiles_are_exchanged():
    """Shapes of both sides, measured with 74 pairs of CTAs: one accumulator over all ranks' k where that fills the chip, else the ranks' own products and an exchange."""
    from piccl_b200 import _native as N
    f = N.lib().piccl_test_tp_width
    exchanged = [(8, 1024, 256, 4096), (8, 2048, 256, 4096), (8, 3072, 256, 3776), (8, 1024, 768, 2560), (8, 2048, 1280, 1664), (4, 512, 512, 4096), (4, 1024, 1024, 4096), (3, 384, 512, 4096)]
    read = [(8, 8192, 8192, 3584), (8, 1024, 8192, 4096), (8, 1024, 4096, 2048), (8, 1024, 512, 960), (8, 3072, 1024, 4096), (8, 1024, 2560, 3712), (4, 512, 2048, 4096), (4, 1024, 512, 1728),
            (3, 1152, 512, 2048), (2, 512, 256, 4096), (2, 4096, 4096, 2048), (8, 1024, 256, 256)]
    assert all(f(0, *s, 74) == 0 for s in exchanged)
    assert all(f(0, *s, 74) in (64, 128, 256) for s in read)
    assert all(f(1, *s, 74) in (64, 128, 256) for s in exchanged + read)      # an all-gather's product sums no more than its own k either way
