"""Which SM and which page lies on which die, told from latencies (no GPU: made-up figures)."""
import ctypes as C

import numpy as np
import pytest

GROUPS, GROUP_PAGES, POOL, SMS, PROBE = 8, 124, 2304, 256, 8


def measured(rng, first, second, home_of_page, by=None):
    """Latencies as an SM of one die has them to pages of its own (near) and of the other, within 12 %; the SMs' dies."""
    die = np.full(SMS, -1)
    present = np.sort(rng.permutation(SMS)[:first + second])
    die[present] = 0
    die[rng.permutation(present[1:])[:second]] = 1                    # the first SM that is there names die 0

    def cycles(sm, home):
        near = np.where(die[sm] == home, 1.0, 2.2)
        return (700.0 * near * rng.uniform(0.94, 1.06, size=near.shape)).astype(np.uint32)

    homes = np.array([0, 1, 1, 0, 1, 0, 0, 1])
    of_sm = np.zeros((SMS, PROBE), dtype=np.uint32)
    for sm in present:
        of_sm[sm] = cycles(sm, homes)
    run = -(-POOL // len(present))
    by = present[np.arange(POOL) // run] if by is None else present[by]
    return of_sm, cycles(by, home_of_page), by.astype(np.uint32), die


def sort(q3t, of_sm, of_page, by, sms):
    lib = q3t.library()
    lib.q3t_test_sort_chain_places.argtypes = [C.c_void_p] * 3 + [C.c_int32] + [C.c_void_p] * 2
    die, pages = np.full(SMS, 9, dtype=np.uint8), np.full((GROUPS, GROUP_PAGES), 1 << 30, dtype=np.uint32)
    groups = lib.q3t_test_sort_chain_places(*(np.ascontiguousarray(a).ctypes.data for a in (of_sm, of_page, by)), sms,
                                            die.ctypes.data, pages.ctypes.data)
    if groups == GROUPS:
        assert (die == 9).all() and (pages == 1 << 30).all()          # any place will do
    return groups, die, pages


PARITY = np.array([bin(p).count("1") % 2 for p in range(POOL)])


@pytest.mark.parametrize("first,second,groups", [(74, 74, 4), (70, 78, 4), (78, 70, 4), (60, 88, 4), (88, 50, 5), (40, 108, 3), (64, 64, 4), (130, 18, 7)])
@pytest.mark.parametrize("homes", ["parity", "low bit", "high bit of sixteen"])
def test_dies_are_told_apart(q3t, first, second, groups, homes):
    pages_at = np.arange(POOL)
    home = {"parity": PARITY, "low bit": pages_at % 2, "high bit of sixteen": pages_at // 8 % 2}[homes]
    of_sm, of_page, by, die = measured(np.random.default_rng(first), first, second, home)
    need = max(groups, GROUPS - groups) * GROUP_PAGES
    got, die_of_sm, pages = sort(q3t, of_sm, of_page, by, first + second)
    assert got == groups and need <= POOL // 2
    assert (die_of_sm[die >= 0] == die[die >= 0]).all() and die_of_sm.max() == 1
    assert len(np.unique(pages)) == GROUPS * GROUP_PAGES and pages.max() < POOL
    for g in range(GROUPS):
        assert (home[pages[g]] == (0 if g < groups else 1)).all()


def test_where_it_cannot_be_told(q3t):
    rng = np.random.default_rng(1)
    of_sm, of_page, by, _ = measured(rng, 148, 0, PARITY)             # one die
    assert sort(q3t, of_sm, of_page, by, 148)[0] == GROUPS
    of_sm, of_page, by, _ = measured(rng, 74, 74, PARITY)
    assert sort(q3t, of_sm, of_page, by, 148)[0] == 4
    assert sort(q3t, of_sm, of_page, by, 149)[0] == GROUPS            # an SM on which the probe did not run
    few = np.arange(POOL) % 8 == 0                                    # 288 pages of one die, 496 are needed
    of_sm, of_page, by, _ = measured(rng, 74, 74, few)
    assert sort(q3t, of_sm, of_page, by, 148)[0] == GROUPS


def test_pages_of_an_sm_that_saw_one_band_count_for_nothing(q3t):
    """Two SMs saw pages of one die only, their own or the other: whose they are cannot be told, and no group gets them."""
    rng = np.random.default_rng(2)
    by = np.arange(POOL) // 16
    home = PARITY.copy()
    for lone, where in ((5, 0), (90, 1)):
        home[by == lone] = where
    of_sm, of_page, by, die = measured(rng, 74, 74, home, by)
    groups, _, pages = sort(q3t, of_sm, of_page, by, 148)
    assert groups == 4
    lone = np.unique(by)[[5, 90]]
    assert not np.isin(by[pages], lone).any()
    for g in range(GROUPS):
        assert (home[pages[g]] == (0 if g < groups else 1)).all()
