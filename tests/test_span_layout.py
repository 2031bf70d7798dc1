"""Host-side checks of the batched path's spans (jellyfih_b200/csrc/jf_span.cu),
restated here in Python: the groups and window size jf_span_setup picks, the
cuts of span_cut_kernel for any row costs, and the cuts by window size alone.
Every layout has to cover each instance's rows once and in order with bands of
at least four rows, so that the overlaps of a band's two cuts stay apart and
only neighbours share rows, and every CTA's windows have to fit."""
import numpy as np
import pytest

K_HALO, K_MIN_ROWS, K_MAX_SEG, K_OVERLAP = 4, 4, 8, 4
HARD = (227 * 1024 - 3072) // 20
SOFT = (96 * 1024) // 20
N_SM = 148


def setup(shapes, n_sm=N_SM):
    """jf_span_setup: (groups of (m0, m1, row0, rows, n_cta), window nodes), None when ineligible."""
    rowoff = np.concatenate([[0], np.cumsum([ny for _, ny in shapes])]).tolist()
    M, nx_max = len(shapes), max(nx for nx, _ in shapes)
    n_groups = 1
    while True:
        groups, need, m = [], 0, 0
        for k in range(n_groups):
            if m >= M:
                break
            m0 = m
            upto = rowoff[M] * (k + 1) // n_groups
            m += 1
            while m < M and (k == n_groups - 1 or rowoff[m + 1] <= upto):
                m += 1
            rows = rowoff[m] - rowoff[m0]
            n_cta = max(1, min(n_sm, rows // K_MIN_ROWS))
            nodes = sum(nx * ny for nx, ny in shapes[m0:m])
            need = max(need, nodes // n_cta + (2 if m - m0 > 1 else 1) * K_HALO * nx_max)
            groups.append((m0, m, rowoff[m0], rows, n_cta))
        assert groups[-1][1] == M or n_groups > 0
        if need <= SOFT:
            break
        n_groups = n_groups + 1 if n_groups < 8 else n_groups * 2
        if n_groups > M:
            break
    assert groups[0][0] == 0 and groups[-1][1] == M
    assert all(a[1] == b[0] for a, b in zip(groups, groups[1:]))
    cap = min(max(need + need * 3 // 5, (4 * K_MIN_ROWS + K_HALO) * nx_max), HARD)
    for tries in (cap, HARD):
        falls = [fill_cuts(shapes, g, rowoff, tries) for g in groups]
        if all(f is not None for f in falls):
            return groups, tries, rowoff, falls
    return None


def fill_cuts(shapes, g, rowoff, cap):
    cuts, room, left = [0], cap, K_MAX_SEG
    for m in range(g[0], g[1]):
        nx, ny = shapes[m]
        b, y = rowoff[m] - g[2], 0
        while y < ny:
            rows = min(room // nx - K_HALO, ny - y) if left > 0 else 0
            if 0 < ny - y - rows < K_MIN_ROWS:
                rows = ny - y - K_MIN_ROWS
            if rows < K_MIN_ROWS:
                if cuts[-1] == b + y:
                    return None
                cuts.append(b + y)
                room, left = cap, K_MAX_SEG
                continue
            room -= (rows + K_HALO) * nx
            left -= 1
            y += rows
    if len(cuts) > g[4]:
        return None
    return cuts + [g[3]] * (g[4] + 1 - len(cuts))


def cut(shapes, g, rowoff, cap, cost):
    """span_cut_kernel's cuts, None where it falls back."""
    m, R, n = g[0], g[3], g[4]
    pre = np.cumsum(cost)
    total = int(pre[-1])
    at_cost = pre - np.asarray(cost) // 2
    ideal = [0] + [int(np.searchsorted(at_cost, total * q // n, side="left")) for q in range(1, n)]
    prev, cuts = 0, []
    for q in range(1, n + 1):
        if prev >= R:
            break
        y = ideal[q] if q < n else R
        while prev >= rowoff[m + 1] - g[2]:
            m += 1
        y = max(y, prev + K_MIN_ROWS)
        at, mm, room, left = prev, m, cap, K_MAX_SEG
        while True:
            bb, ee, nx = rowoff[mm] - g[2], rowoff[mm + 1] - g[2], shapes[mm][0]
            stop = min(y, ee)
            if stop < ee and ee - stop < K_MIN_ROWS:
                stop = ee
            if stop < ee and stop - bb < K_MIN_ROWS:
                stop = at if at > prev else bb + K_MIN_ROWS
            if left == 0:
                stop = at
            if stop > at and (stop - at + K_HALO) * nx > room:
                stop = at + room // nx - K_HALO
                if ee - stop < K_MIN_ROWS:
                    stop = ee - K_MIN_ROWS
                if stop - at < K_MIN_ROWS:
                    stop = at
            if stop > at:
                room -= (stop - at + K_HALO) * nx
                left -= 1
            at = stop
            if at < ee or at >= y or at >= R:
                break
            mm += 1
        if at <= prev:
            return None
        cuts.append(prev)
        prev = at
    return None if prev < R else cuts + [R] * (n + 1 - len(cuts))


def check(shapes, g, rowoff, cap, cuts):
    assert cuts[0] == 0 and cuts[-1] == g[3] and len(cuts) == g[4] + 1
    done = {m: 0 for m in range(g[0], g[1])}
    last = None
    for c, (lo, hi) in enumerate(zip(cuts, cuts[1:])):
        assert lo <= hi
        at, nodes, segs = lo, 0, 0
        while at < hi:
            m = int(np.searchsorted(np.asarray(rowoff) - g[2], at, side="right")) - 1
            b, e = rowoff[m] - g[2], rowoff[m + 1] - g[2]
            stop = min(hi, e)
            first, end, ny = at - b, stop - b, e - b
            assert done[m] == first and end - first >= K_MIN_ROWS
            if first > 0:  # the lower neighbour is the CTA before, this the CTA's first band
                assert last == c - 1 and segs == 0 and first - 1 >= 0 and first + 2 < ny
            done[m] = end
            nodes += (end - first + K_HALO) * shapes[m][0]
            segs += 1
            last = c
            at = stop
        assert nodes <= cap and segs <= K_MAX_SEG
    assert all(done[m] == shapes[m][1] for m in done)


BATCHES = [[(128, 128)], [(128, 128)] * 2, [(128, 128)] * 8, [(128, 128)] * 16, [(128, 128)] * 32,
           [(128, 256)] * 8, [(128, 128)] * 48 + [(128, 256)] * 16, [(64, 64)] * 256, [(32, 32)], [(8, 8)] * 3,
           [(8, 9)] * 100, [(80, 112), (96, 96), (128, 256)], [(128, 128)] * 300, [(1000, 40)], [(37, 1024)],
           [(256, 256)] * 40, [(8, 1024)] * 5]


@pytest.mark.parametrize("shapes", BATCHES, ids=lambda s: f"{len(s)}x{s[0][0]}x{s[0][1]}")
def test_spans_cover_the_rows_and_fit(shapes):
    groups, cap, rowoff, falls = setup(shapes)
    rng = np.random.default_rng(len(shapes))
    for g, fall in zip(groups, falls):
        check(shapes, g, rowoff, cap, fall)
        fell = 0
        for trial in range(24):
            kind, R = trial % 4, g[3]
            if kind == 0:
                cost = rng.integers(0, 5000, R)
            elif kind == 1:
                cost = np.zeros(R, np.int64)
                cost[rng.integers(0, R, 3)] = 10 ** 6
            elif kind == 2:
                cost = np.zeros(R, np.int64)
            else:
                cost = np.where(np.arange(R) % 128 < 64, 4000, 0)
            got = cut(shapes, g, rowoff, cap, cost.astype(np.int64) + 40)
            fell += got is None
            if got is not None:
                check(shapes, g, rowoff, cap, got)
            if kind == 2:
                assert got is not None  # equal costs never fall back


def test_spans_use_every_sm_of_a_full_batch():
    for shapes in ([(128, 128)] * 32, [(128, 128)] * 16, [(128, 256)] * 8):
        groups, cap, rowoff, _ = setup(shapes)
        assert len(groups) == 1 and groups[0][4] == N_SM
        got = cut(shapes, groups[0], rowoff, cap, np.full(groups[0][3], 2000))
        assert len(set(got)) == N_SM + 1


@pytest.mark.parametrize("shapes", [[(8, 8)] * 2000, [(2000, 8)]])
def test_batches_that_do_not_suit_spans_keep_the_clusters(shapes):
    assert setup(shapes) is None
