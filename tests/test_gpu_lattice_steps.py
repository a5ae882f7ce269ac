"""GPU parity of the lattice cursor's steps: counts around multiples of four,
codes of up to 13 bits (L = 8192, rare symbols in a row), and runs of zero-bit
codewords longer than an entry can count (255).  Integer work: the tolerance
is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _symbols(kind, n, rng):
    if kind == "flat":      # every byte value equally rare: the longest codes
        return rng.integers(0, 256, n).astype(np.uint8)
    if kind == "rare":      # runs of rare symbols inside one frequent symbol
        s = np.zeros(n, np.uint8)
        at = rng.random(n) < 0.02
        s[at] = rng.integers(1, 256, int(at.sum()))
        for i in range(0, n - 8, 997):
            s[i: i + 8] = np.arange(200, 208)
        return s
    s = np.zeros(n, np.uint8)   # "runs": one symbol but for one in 3000
    s[rng.random(n) < 1 / 3000] = 7
    if n > 1:
        s[n // 2] = 9
    return s


@pytest.mark.parametrize("L", [64, 1024, 4096, 8192])
@pytest.mark.parametrize("kind", ["flat", "rare", "runs"])
def test_steps(mg, oracle_lib, kind, L):
    from multians_gb300.decoder import decode
    O = oracle_lib
    rng = np.random.default_rng(L + len(kind))
    for n in (2, 3, 4, 5, 7, 8, 9, 255, 4097, 70_003, 1_500_001):
        sym = _symbols(kind, n, rng)
        if L < 256:
            sym = (sym % 16).astype(np.uint8)
        st = O.encode(sym, L)
        want = O.decode_seq(st)
        if not np.array_equal(want, sym[::-1]):
            continue   # not decodable: the sequential decode runs past the units as well
        for so in (False, True):
            got = decode(st.units, st.n_units, n, st.table, st.first_state, st.first_bit, L,
                         source_order=so).cpu().numpy()
            assert np.array_equal(got, want[::-1] if so else want), (n, so)
