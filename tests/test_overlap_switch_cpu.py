"""The switch for overlapping launches (host side only)."""
import threading


def test_a_threads_own():
    from art_b200.ops import paged

    seen = []
    before = paged.set_pdl(2)

    def other():
        seen.append(paged.set_pdl(1))
        seen.append(paged.set_pdl(0))

    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert seen == [0, 1]
    assert paged.set_pdl(before) == 2


def test_products_overlap_their_own_kind():
    """1 and 2: products with tiles of one CTA and of CTA pairs, whose tensor-memory allocations must not meet."""
    from art_b200.ops import _lib, paged

    overlaps = _lib.kernels().artb_product_overlaps
    for mode in (1, 2):
        before = paged.set_pdl(mode)
        # the first product after the switch is set follows whatever ran before it
        assert [overlaps(c) for c in (1, 1, 1, 2, 2, 1, 2, 2, 1, 1)] == [0, 1, 1, 0, 1, 0, 0, 1, 0, 1]
        paged.set_pdl(mode)
        assert overlaps(1) == 0
        assert paged.set_pdl(before) == mode
    before = paged.set_pdl(0)
    assert not any(overlaps(c) for c in (1, 1, 2, 2))
    paged.set_pdl(before)
