"""The exchange tags of the region solve after a solve that a timed-out wait
ended. CTAs in a row exchange epoch-tagged words as k_sor_tb does (two lists by
parity, a CTA publishes epoch e and needs its neighbours' words of e before
e + 1); one of them stops for good, the others go on until a word is missing.
The tag base that csrc/ws_sor_tags.h then leaves must be one from which no later
epoch waits for a tag that some list still holds."""
import ctypes
import os
import subprocess

import pytest

from conftest import PKG


@pytest.fixture(scope="module")
def next_base(tmp_path_factory):
    d = tmp_path_factory.mktemp("tags")
    src, so = d / "tags.c", d / "tags.so"
    src.write_text('#include "%s"\nunsigned next_base(unsigned t, unsigned e, int a, int n) '
                   '{ return tb_next_tag_base(t, e, a, n); }\n' % os.path.join(PKG, "csrc", "ws_sor_tags.h"))
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    L = ctypes.CDLL(str(so))
    L.next_base.argtypes = [ctypes.c_uint32, ctypes.c_uint32, ctypes.c_int, ctypes.c_int]
    L.next_base.restype = ctypes.c_uint32
    return L.next_base


def _solve(lists, tag0, epochs, stuck, stuck_at, links):
    """One solve over the CTAs' lists[cta][parity]; CTA `stuck` publishes nothing
    after epoch stuck_at (None: nobody). Returns CTA 0's epochs and whether it
    waited in vain."""
    P = len(lists)
    done = [0] * P
    moved = True
    while moved:
        moved = False
        for p in range(P):
            if done[p] == epochs or (p == stuck and done[p] == stuck_at):
                continue
            e = done[p]
            if e and not all(lists[n][e & 1] == (tag0 + e) % 2 ** 32 for n in links[p]):
                continue
            lists[p][(e + 1) & 1] = (tag0 + e + 1) % 2 ** 32
            done[p] += 1
            moved = True
    return done[0], done[0] < epochs


@pytest.mark.parametrize("tag0", [0, 7, 2 ** 32 - 9])
@pytest.mark.parametrize("apart", [False, True])
def test_no_stale_word_matches_after_an_aborted_solve(next_base, tag0, apart):
    P, iters = 12, 20
    links = [[n for n in (p - 1, p + 1) if 0 <= n < P] for p in range(P)]
    if apart:                                    # two groups that share no halo: the second runs to its end
        links[5], links[6] = [4], [7]
    for stuck in range(6 if apart else P):
        for at in range(0, 8):
            lists = [[0, 0] for _ in range(P)]
            ran, aborted = _solve(lists, tag0, iters, stuck, at, links)
            assert aborted
            base = next_base(tag0, ran, 1, iters)
            for p in range(P):
                for parity in (0, 1):
                    ahead = (lists[p][parity] - base) % 2 ** 32
                    assert lists[p][parity] == 0 or not (1 <= ahead < 2 ** 31 and ahead % 2 == parity), (stuck, at, p)


def test_tags_count_on_without_a_gap_after_a_whole_solve(next_base):
    """A solve that ended advances by its epochs: the tags last for 2^32 of them."""
    lists = [[0, 0] for _ in range(3)]
    ran, aborted = _solve(lists, 5, 9, None, None, [[1], [0, 2], [1]])
    assert (ran, aborted) == (9, False)
    assert next_base(5, ran, 0, 1000) == 5 + 9 + 1
