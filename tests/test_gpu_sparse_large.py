"""The sparse map's large primes (GPU): rows so short that nearly every sieving
prime from 2^20 on misses them, at the heights where its quotient is smallest
and largest; every bit against Miller-Rabin."""
import pytest

import gbc
import oracle

pytestmark = pytest.mark.gpu
M = 30030


@pytest.mark.parametrize("height", [3 * 10**12, 10**16, 2**63, gbc.MAX_LIMIT - 10**9])
def test_short_rows_bit_exact(height):
    n0, dl = height - height % M, 64
    with gbc.Sparse(limit=n0 + M * dl, dlt_log2=12, pmax=1_000_000) as sp:
        rows = sp.map(n0, dl)
        q0 = n0 - M * sp.tb
        for k in range(sp.K):
            for t in range(dl + sp.tb):
                q = q0 + sp.residues[k] + M * t
                assert ((rows[k][t >> 5] >> (t & 31)) & 1) == oracle.is_prime(q), (k, t)
