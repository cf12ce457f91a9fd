"""The committed lookup tables are the generator's output."""

import os
import re
import sys

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "isoext_gb300", "csrc")
sys.path.insert(0, CSRC)
import gen_luts  # noqa: E402


def test_luts_header_is_current():
    with open(os.path.join(CSRC, "luts.h")) as fh:
        assert fh.read() == gen_luts.render()


def test_luts_counts():
    nag = gen_luts.expand(gen_luts.NAGAE, reflect=False)
    lor = gen_luts.expand(gen_luts.LORENSEN, reflect=True)
    assert max(len(t) for t in nag) == 5 and max(len(t) for t in lor) == 4
    st = gen_luts.edge_status(nag)
    assert st[0] == 0 and st[255] == 0 and all(st[i] for i in range(1, 255))


def _ref_table(path, name):
    s = open(path).read()
    i = s.index(name)
    body = re.sub(r"//.*", "", s[s.index("{", i) + 1: s.index("}", i)])
    return [int(x, 0) for x in re.findall(r"-?0b[01]+|-?\d+", body)]


def test_luts_equal_reference_fixture():
    """The generated tables equal the reference's, as stored by make_golden.py luts."""
    import numpy as np

    ref = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "luts_ref.npz"))
    nag = gen_luts.flat(gen_luts.expand(gen_luts.NAGAE, False), 15)
    lor = gen_luts.flat(gen_luts.expand(gen_luts.LORENSEN, True), 12)
    assert nag == ref["nagae_tri"].tolist()
    assert lor == ref["lorensen_tri"].tolist()
    assert gen_luts.edge_status(gen_luts.expand(gen_luts.NAGAE, False)) == ref["edge_status"].tolist()


def test_luts_equal_reference_tables():
    """Same, read live from an isoext checkout named by $ISOEXT_REFERENCE."""
    ref = os.environ.get("ISOEXT_REFERENCE")
    if not ref or not os.path.isdir(os.path.join(ref, "include")):
        pytest.skip("ISOEXT_REFERENCE does not name an isoext checkout")
    nag = gen_luts.flat(gen_luts.expand(gen_luts.NAGAE, False), 15)
    lor = gen_luts.flat(gen_luts.expand(gen_luts.LORENSEN, True), 12)
    assert nag == _ref_table(os.path.join(ref, "include/mc/nagae.cuh"), "tri_table[]")
    assert lor == _ref_table(os.path.join(ref, "include/mc/lorensen.cuh"), "tri_table[]")
    st = gen_luts.edge_status(gen_luts.expand(gen_luts.NAGAE, False))
    assert st == _ref_table(os.path.join(ref, "src/shared_luts.cu"), "edge_status_table[edge_table_size]")


def test_packed_triangle_lists_match_tables():
    for method, (table, width) in enumerate([(gen_luts.NAGAE, 15), (gen_luts.LORENSEN, 12)]):
        cases = gen_luts.expand(table, reflect=method == 1)
        flat = gen_luts.flat(cases, width)
        packed = gen_luts.packed(cases)
        for c in range(256):
            v = packed[c]
            n = v >> 60
            edges = [(v >> (4 * i)) & 15 for i in range(3 * n)]
            row = [e for e in flat[c * width:(c + 1) * width] if e >= 0]
            assert edges == row and n == len(cases[c])


def test_one_polygon_cells_have_two_triangles_less_than_crossed_edges():
    """The MC count's rule (word_faces): outside the cases with a face whose diagonal
    corners pair up, or two opposite corners against the other six, both tables
    have (crossed edges - 2) triangles."""
    edges = [(a, a | d) for a in range(8) for d in (1, 2, 4) if not a & d]
    faces = [(0, 1, 3, 2), (4, 5, 7, 6), (0, 1, 5, 4), (2, 3, 7, 6), (0, 2, 6, 4), (1, 3, 7, 5)]
    checked = 0
    for table, reflect in ((gen_luts.NAGAE, False), (gen_luts.LORENSEN, True)):
        for cs, tris in enumerate(gen_luts.expand(table, reflect)):
            c = [(cs >> k) & 1 for k in range(8)]
            many = any(c[a] == c[d] and c[b] == c[e] and c[a] != c[b] for a, b, d, e in faces)
            many |= any(c[i] == c[7 - i] and all(c[k] != c[i] for k in range(8) if k not in (i, 7 - i)) for i in range(4))
            if cs in (0, 255) or many:
                continue
            assert len(tris) == sum(c[a] != c[b] for a, b in edges) - 2, cs
            checked += 1
    assert checked > 200
