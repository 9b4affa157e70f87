"""The index arithmetic of k_poisson_scan (poisson_scan.cu), on CPU: for grids of every size up to
2600 and some larger, alone and in sets of larger runs, every element that a block reads from
another block's vector lies in that block's share of it, and the values about a block's cells
are the ones its E_x needs."""
import pytest

CLUSTER, MAX_THREADS = 8, 512


def _threads(maxn):
    t = 32
    while t < MAX_THREADS and t * CLUSTER * 8 < maxn - 1:
        t *= 2
    return t


def _check(n, maxn):
    m, T = n - 1, _threads(maxn)
    L = -(-m // (T * CLUSTER))
    share = [max(0, min(T * L, m - r * T * L)) for r in range(CLUSTER)]
    assert sum(share) == m and L <= -(-(maxn - 1) // (T * CLUSTER))  # the launch's shared memory holds it

    def remote(g):
        r = g // (T * L)
        assert 0 <= r < CLUSTER and 0 <= g - r * T * L < share[r], (n, maxn, g)

    for g in (0, 1, m - 1):
        remote(g)
    for rank in range(CLUSTER):
        cnt, g0 = share[rank], rank * T * L
        p0, p1 = (0 if rank == 0 else g0 + 1), g0 + cnt + 1
        halo = {}
        for lane in range(9 if cnt > 0 else 5):
            pe = (lane + 1 if lane < 2 else n - 5 + lane if lane < 5 else p0 - 7 + lane if lane < 7 else p1 - 7 + lane)
            want = pe % n
            pe = pe + n if pe < 0 else pe - n if pe >= n else pe
            assert 0 <= pe < n and pe == want, (n, maxn, rank, lane)
            if pe > 0:
                remote(pe - 1)
            if lane >= 5:
                halo[lane - 5] = pe
        if cnt > 0:
            assert [halo[k] for k in range(4)] == [(p0 - 2) % n, (p0 - 1) % n, p1 % n, (p1 + 1) % n]
            assert p1 <= n


@pytest.mark.parametrize("maxn", [0, 4096, 4098, 16384, 196608])
def test_remote_reads_stay_in_their_blocks(maxn):
    for n in list(range(5, 2600)) + [3000, 4095, 4096, 4097, 4098, 8192, 12345, 16384, 65536, 196609]:
        if maxn == 0 or n <= maxn:
            _check(n, max(n, maxn))
