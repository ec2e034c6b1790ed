"""Device bytes of a Krylov handle as admission and placement count them (rr_footprint) against
the buffers a handle allocates: the CSR copies, the blocks and preconditioner forms, the sequence,
the sums of both Gram terms and the slots of a resident run."""
import pytest

import rust_rank_b200 as rr

RUN_APPS = 512   # applications of one resident run, at most
REPLICAS = 8     # of the Gram sums of the passes


def held(m, n, nnz, b):
    B = 4 if b <= 4 else 8 if b <= 8 else 16 if b <= 16 else 32
    pairs = B * (B + 1) // 2
    csr = 2 * 8 * nnz + 4 * (m + n + 2) + 4 * (m + n)  # entries and offsets twice, both renumberings
    blocks = 4 * B * (2 * n + m)
    forms = 4 * (2 * m + 4 * n + 4)
    seq = 4 * (b * (b + 1) // 2) * (rr.default_max_nlen(m, n, b) + 1)
    gram = 8 * REPLICAS * 2 * pairs
    runs = 8 * 2 * RUN_APPS * pairs if B <= 16 else 0
    return csr + blocks + forms + seq + gram + runs


@pytest.mark.parametrize("b", [1, 4, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("m,n", [(1, 1), (40, 30), (1000, 800), (20000, 15000), (200000, 150000)])
def test_footprint_covers_what_a_handle_holds(m, n, b):
    assert rr.footprint(m, n, 6 * m, b) >= held(m, n, 6 * m, b)
