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
