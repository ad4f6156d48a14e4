"""The reference-order libm mode prices two options at a time with its own
division, square root and reciprocal while every operand is inside the range
these round correctly in, and one by one otherwise.  At and beyond the edges
of that range an option in a book gets the bits it gets alone (a book of one
option is priced one by one)."""
import dataclasses
import itertools

import numpy as np
import pytest

from p3arsec_gb300 import books

pytestmark = pytest.mark.gpu

LO, HI = np.float32(2.0 ** -30), np.float32(2.0 ** 30)
EDGES = [np.float32(x) for x in (0.0, 1e-42, np.nextafter(LO, np.float32(0)), LO, 1.0,
                                 np.nextafter(np.float32(1), np.float32(0)), HI,
                                 np.nextafter(HI, np.float32(np.inf)), np.inf, np.nan, -1.0)]


def edge_book():
    rows = []
    for i, j in itertools.combinations(range(6), 2):
        for a, b in itertools.product(EDGES, repeat=2):
            row = [np.float32(x) for x in (100, 90, 0.05, 0.3, 0.5)] + [len(rows) & 1]
            row[i] = a
            if j < 5:
                row[j] = b
            else:
                row[2] = np.float32(174) * b  # -r t = -87 at b = 1
            rows.append(row)
    return rows


def test_bits_at_the_edges_of_the_paired_range(gpu_ctx):
    rows = edge_book()
    # an edge case in one place of each pair, an ordinary option in the other;
    # a book of this length is priced four options to a thread
    m = 2 * len(rows)
    book = books.generate(1 << 15, seed=5, dist="tails")
    cols = [np.array(getattr(book, f.name)) for f in dataclasses.fields(books.Book)][:6]
    for i, row in enumerate(rows):
        for c, x in zip(cols, row):
            c[2 * i + (i >> 1 & 1)] = x
    got = gpu_ctx.price_book(books.Book(*cols), num_runs=1, mode="libm_ref")[:m]
    alone = np.concatenate([gpu_ctx.price_book(books.Book(*[c[i:i + 1] for c in cols]),
                                               num_runs=1, mode="libm_ref") for i in range(m)])
    same = (got.view(np.uint32) == alone.view(np.uint32)) | (np.isnan(got) & np.isnan(alone))
    bad = np.flatnonzero(~same)
    assert bad.size == 0, [([c[i] for c in cols], got[i], alone[i]) for i in bad[:5]]
