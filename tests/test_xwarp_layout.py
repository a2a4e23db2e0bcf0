"""Buffer layout of the warp-per-unit x pass (mpc_kernels.cuh XWarp): host-side checks of the padded
exchange positions, for rows of 128, 256 and 512."""
import pytest

CFG = {512: (5, 2, 544), 256: (4, 1, 272), 128: (3, 1, 152)}   # pad shift, pad, row stride


def _wavefronts(elems, width=8):
    """128-byte wavefronts of one warp-wide access to elements of `width` bytes."""
    per = 128 // width
    total = 0
    for g in range(0, 32, per):
        banks = {}
        for e in elems[g:g + per]:
            for w in range(e * width // 4, (e + 1) * width // 4):
                banks.setdefault(w % 32, set()).add(w)
        total += max(len(v) for v in banks.values())
    return total


@pytest.mark.parametrize("nx", sorted(CFG))
def test_exchange_positions(nx):
    sh, pad, rs = CFG[nx]
    idx = lambda p: p + (p >> sh) * pad  # noqa: E731
    m, rows = nx // 16, 512 // nx
    assert len({idx(p) for p in range(nx)}) == nx and idx(nx - 1) < rs and rs * 8 % 16 == 0 and m == 1 << sh
    outer, inner = set(), set()
    for q in range(16):
        nat = [(t // m) * rs + t % m + m * q for t in range(32)]            # natural positions (load, store)
        exch = [(t // m) * rs + t % m + idx(m * q) for t in range(32)]      # the outer stage's exchange side
        assert exch == [(t // m) * rs + idx(t % m + m * q) for t in range(32)]
        assert _wavefronts(nat) == 2 and _wavefronts(exch) == 2
        outer |= set(exch)
        if nx == 512:
            e = [idx(32 * (t >> 1)) + (t & 1) + 2 * q for t in range(32)]
            assert e == [idx(32 * (t >> 1) + (t & 1) + 2 * q) for t in range(32)]
            assert _wavefronts(e, 16) == 4                                   # the factors, 16 bytes each
        elif nx == 256:
            e = [(t // m) * rs + idx(16 * (t % m)) + q for t in range(32)]
            assert e == [(t // m) * rs + idx(16 * (t % m) + q) for t in range(32)]
            assert _wavefronts([x % rs for x in e], 16) == 4
        else:
            h, i = divmod(q, 8)
            e = [(t // m) * rs + idx(8 * (t % m + 8 * h)) + i for t in range(32)]
            assert e == [(t // m) * rs + idx(8 * (t % m + 8 * h) + i) for t in range(32)]
        assert _wavefronts(e) == 2
        inner |= set(e)
    assert outer == inner == {r * rs + idx(p) for r in range(rows) for p in range(nx)}


def test_plane_in_shared_memory():
    """The whole-plane kernel's rows (PlaneS): aligned, disjoint with room for the exchange positions, and
    every pass of the y and the x part at the minimum of two wavefronts."""
    n, m, lpu, rstr = 64, 4, 8, 88
    at = lambda y: y * rstr + 4 * (y >> 1)  # noqa: E731
    idx = lambda p: p + (p >> 2)  # noqa: E731
    assert all(at(y) * 8 % 16 == 0 and at(y) + idx(n - 1) < (at(y + 1) if y < n - 1 else at(n - 1) + rstr) for y in range(n))
    lanes = range(32)
    jx, r = [t & 3 for t in lanes], [t >> 2 for t in lanes]
    c, jy = [t & (lpu - 1) for t in lanes], [t // lpu for t in lanes]
    assert len(set(zip(jx, r))) == len(set(zip(jy, c))) == 32
    for u in range(n // lpu):
        seen = [set() for _ in range(4)]
        for q in range(16):
            col = [at(jy[t] + m * q) + u * lpu + c[t] for t in lanes]
            assert col == [at(jy[t]) + at(m * q) - at(0) + u * lpu + c[t] for t in lanes]
            nat = [at(u * lpu + r[t]) + jx[t] + m * q for t in lanes]
            exch = [at(u * lpu + r[t]) + idx(jx[t] + m * q) for t in lanes]
            assert exch == [at(u * lpu + r[t]) + jx[t] + idx(m * q) for t in lanes]
            h, i = divmod(q, m)
            by = [at(m * (jy[t] + m * h) + i) + u * lpu + c[t] for t in lanes]
            assert by == [at(m * (jy[t] + m * h)) + at(i) + u * lpu + c[t] for t in lanes]
            bx = [at(u * lpu + r[t]) + idx(m * (jx[t] + m * h) + i) for t in lanes]
            assert bx == [at(u * lpu + r[t]) + idx(m * (jx[t] + m * h)) + i for t in lanes]
            for e in (col, nat, exch, by, bx):
                assert _wavefronts(e) == 2, (n, u, q)
            for k, e in enumerate((col, by, exch, bx)):
                seen[k] |= set(e)
        assert seen[0] == seen[1] == {at(y) + x for y in range(n) for x in range(u * lpu, (u + 1) * lpu)}
        assert seen[2] == seen[3] == {at(y) + idx(x) for y in range(u * lpu, (u + 1) * lpu) for x in range(n)}
