"""Build step: generate the marching-cubes lookup tables header.

The case tables used by the reference (include/tables.h: edgeTable[256] at :22,
triTable[256][16] at :61 with X=255 as terminator, numVertsTable[256] at :323,
nrOfTriangles[256] at :584, offsets3[72] at :588) are the classic Lorensen/Bourke tables
in the reference's own edge numbering.  That file carries a third-party licence header,
so its text is not committed here: this script reads the numbers from the reference
checkout at build time and writes them, in this project's own format, to
csrc/generated/kf_mc_tables.inc (git-ignored; it ships beside the built libraries).

Usage: python gen_mc_tables.py [path/to/tables.h] [out.inc]

The reference's tables.h is looked for, in order, at: the first argument; $KF_MC_TABLES_H
(a path to tables.h); $KF_REFERENCE_DIR/include/tables.h (a checkout of the reference);
baseline/_ref/include/tables.h under the repository root; include/tables.h of a checkout
named `reference` beside the repository.  When none exists, a previously generated
header is kept; with neither, the tables are derived from the cube's geometry (derive()):
the same corner and edge numbering, edge masks and triangle counts, with this project's own
choice of diagonals inside each polygon.
"""
from __future__ import annotations

import os
import re
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(os.path.dirname(HERE))
DEFAULT_OUT = os.path.join(HERE, "generated", "kf_mc_tables.inc")


def candidate_sources() -> list[str]:
    """Where the reference's tables.h may be, in the order they are tried."""
    c = []
    if os.environ.get("KF_MC_TABLES_H"):
        c.append(os.environ["KF_MC_TABLES_H"])
    if os.environ.get("KF_REFERENCE_DIR"):
        c.append(os.path.join(os.environ["KF_REFERENCE_DIR"], "include", "tables.h"))
    c.append(os.path.join(REPO, "baseline", "_ref", "include", "tables.h"))
    c.append(os.path.join(os.path.dirname(REPO), "reference", "include", "tables.h"))
    return c


def _array_body(text: str, name: str) -> str:
    m = re.search(r"\b" + re.escape(name) + r"\s*(\[[^\]]*\])+\s*=\s*\{", text)
    if not m:
        raise ValueError(f"table {name} not found")
    depth, i = 1, m.end()
    while depth:
        c = text[i]
        depth += c == "{"
        depth -= c == "}"
        i += 1
    return text[m.end():i - 1]


def _numbers(body: str) -> list[int]:
    body = re.sub(r"//[^\n]*", "", body)
    body = re.sub(r"/\*.*?\*/", "", body, flags=re.S)
    out = []
    for tok in re.findall(r"0x[0-9a-fA-F]+|\d+|\bX\b", body):
        out.append(255 if tok == "X" else int(tok, 0))
    return out


def parse(path: str) -> dict[str, list[int]]:
    with open(path, "r", encoding="latin-1") as f:
        text = f.read()
    tabs = {
        "edge": _numbers(_array_body(text, "edgeTable")),
        "tri": _numbers(_array_body(text, "triTable")),
        "nverts": _numbers(_array_body(text, "numVertsTable")),
        "ntri": _numbers(_array_body(text, "nrOfTriangles")),
        "offsets3": _numbers(_array_body(text, "offsets3")),
    }
    want = {"edge": 256, "tri": 4096, "nverts": 256, "ntri": 256, "offsets3": 72}
    for k, n in want.items():
        if len(tabs[k]) != n:
            raise ValueError(f"table {k}: {len(tabs[k])} entries, expected {n}")
    check(tabs)
    return tabs


def check(t: dict[str, list[int]]) -> None:
    """Self-consistency facts of the case tables."""
    for c in range(256):
        row = t["tri"][16 * c:16 * c + 16]
        n = next((i for i, e in enumerate(row) if e == 255), 16)
        assert all(e == 255 for e in row[n:]), c
        assert n == t["nverts"][c] == 3 * t["ntri"][c], c
        mask = 0
        for e in row[:n]:
            assert 0 <= e < 12
            mask |= 1 << e
        assert mask == t["edge"][c], c  # every cut edge is used, no other edge is
    assert sum(t["ntri"]) == 820


# Corners in the classic path's numbering (marchingCubes.cs:142-150) and the corner pairs of
# the 12 edges; a face is its four corners in cyclic order.
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
EDGES = [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7)]
FACES = [(0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (3, 2, 6, 7), (0, 3, 7, 4), (1, 2, 6, 5)]


def _edge(a: int, b: int) -> int:
    return next(e for e, p in enumerate(EDGES) if set(p) == {a, b})


def _segments(case: int) -> list[tuple[int, int]]:
    """The contour on each face, as pairs of cut edges: every run of set corners along the
    face's cycle is cut off by one segment (so two set corners on a diagonal stay separate,
    in both cubes that share the face)."""
    segs = []
    for f in FACES:
        inside = [(case >> c) & 1 for c in f]
        if sum(inside) in (0, 4):
            continue
        for k in range(4):
            if inside[k] and not inside[k - 1]:  # a run of set corners starts here
                j = k
                while inside[(j + 1) % 4]:
                    j = (j + 1) % 4
                segs.append((_edge(f[k - 1], f[k]), _edge(f[j], f[(j + 1) % 4])))
    return segs


def _loops(segs: list[tuple[int, int]]) -> list[list[int]]:
    """The face segments joined into closed polygons, each from its lowest edge."""
    left, loops = list(segs), []
    while left:
        a, b = left.pop(min(range(len(left)), key=lambda i: min(left[i])))
        loop = [min(a, b), max(a, b)]
        while loop[0] != loop[-1]:
            i = next(i for i, s in enumerate(left) if loop[-1] in s)
            s = left.pop(i)
            loop.append(s[1] if s[0] == loop[-1] else s[0])
        loops.append(loop[:-1])
    return loops


def _midpoint(e: int) -> list[float]:
    p, q = (CORNERS[c] for c in EDGES[e])
    return [0.5 * (p[k] + q[k]) for k in range(3)]


def _winding(case: int, loop: list[int]) -> float:
    """Sign of the loop's area vector along its own free-space direction (the sum over its
    edges of clear corner - set corner)."""
    m = [_midpoint(e) for e in loop]
    area, out = [0.0] * 3, [0.0] * 3
    for i, e in enumerate(loop):
        u, v = m[i], m[(i + 1) % len(loop)]
        a, b = EDGES[e]
        s, c = (a, b) if (case >> a) & 1 else (b, a)
        for k in range(3):
            area[k] += u[(k + 1) % 3] * v[(k + 2) % 3] - u[(k + 2) % 3] * v[(k + 1) % 3]
            out[k] += CORNERS[c][k] - CORNERS[s][k]
    return sum(area[k] * out[k] for k in range(3))


def _triangulate(loop: list[int]) -> list[tuple[int, int, int]] | None:
    """Triangles of a polygon whose diagonals never join two edges of one cube face (such a
    diagonal would lie in the face, where the neighbour cube's polygon has its own side)."""
    def allowed(a, b):
        ca, cb = EDGES[a], EDGES[b]
        return not any(set(ca) <= set(f) and set(cb) <= set(f) for f in FACES)

    if len(loop) == 3:
        return [(loop[0], loop[1], loop[2])]
    n = len(loop)
    for k in range(1, n - 1):  # the triangle on the side (loop[0], loop[-1]) and its apex
        if (k > 1 and not allowed(loop[0], loop[k])) or (k < n - 2 and not allowed(loop[k], loop[-1])):
            continue
        lo = _triangulate(loop[:k + 1]) if k > 1 else []
        hi = _triangulate(loop[k:]) if k < n - 2 else []
        if lo is not None and hi is not None:
            return [(loop[0], loop[k], loop[-1])] + lo + hi
    return None


def derive() -> dict[str, list[int]]:
    """The case tables from the cube's geometry: on every face the contour cuts off each run
    of set corners, the face segments close into polygons, each polygon is triangulated and
    wound clockwise seen from the clear (free-space) corners.  offsets3 holds the edges' end
    points with y and z swapped (histoPyramids.cs:27-36)."""
    t = {"edge": [], "tri": [], "nverts": [], "ntri": [], "offsets3": []}
    for case in range(256):
        mask = sum(1 << e for e, (a, b) in enumerate(EDGES) if ((case >> a) ^ (case >> b)) & 1)
        row = []
        for loop in _loops(_segments(case)):
            if _winding(case, loop) > 0:
                loop = [loop[0]] + loop[:0:-1]
            tris = _triangulate(loop)
            if tris is None:
                raise ValueError(f"case {case}: no triangulation of {loop}")
            for tri in tris:
                row += tri
        t["edge"].append(mask)
        t["tri"] += row + [255] * (16 - len(row))
        t["nverts"].append(len(row))
        t["ntri"].append(len(row) // 3)
    for a, b in EDGES:
        for c in (a, b):
            x, y, z = CORNERS[c]
            t["offsets3"] += [x, z, y]
    check(t)
    return t


def emit(t: dict[str, list[int]], out: str) -> None:
    os.makedirs(os.path.dirname(out), exist_ok=True)

    def rows(vals, per):
        return ",\n".join("  " + ", ".join(str(v) for v in vals[i:i + per])
                          for i in range(0, len(vals), per))

    tri = [(-1 if v == 255 else v) for v in t["tri"]]
    src = [
        "/* generated by gen_mc_tables.py at build time; do not edit, do not commit */",
        "#define KF_MC_TABLES_GENERATED 1",
        f"KF_MC_TABLE_QUAL uint16_t kf_mc_edge_table[256] = {{\n{rows(t['edge'], 16)}\n}};",
        f"KF_MC_TABLE_QUAL int8_t kf_mc_tri_table[256 * 16] = {{\n{rows(tri, 16)}\n}};",
        f"KF_MC_TABLE_QUAL uint8_t kf_mc_num_verts[256] = {{\n{rows(t['nverts'], 16)}\n}};",
        f"KF_MC_TABLE_QUAL uint8_t kf_mc_nr_triangles[256] = {{\n{rows(t['ntri'], 16)}\n}};",
        f"KF_MC_TABLE_QUAL uint8_t kf_mc_offsets3[72] = {{\n{rows(t['offsets3'], 6)}\n}};",
        "",
    ]
    tmp = out + ".tmp"
    with open(tmp, "w") as f:
        f.write("\n".join(src))
    os.replace(tmp, out)


def main(argv: list[str]) -> int:
    tried = [argv[1]] if len(argv) > 1 else candidate_sources()
    out = argv[2] if len(argv) > 2 else DEFAULT_OUT
    src = next((p for p in tried if os.path.exists(p)), None)
    if src is None:
        if os.path.exists(out):
            print(f"gen_mc_tables: no tables.h found; keeping existing {out}")
            return 0
        if len(argv) > 1:
            print(f"gen_mc_tables: {argv[1]} was not found", file=sys.stderr)
            return 1
        emit(derive(), out)
        print(f"gen_mc_tables: no tables.h found; derived {out} from the cube's geometry")
        return 0
    emit(parse(src), out)
    print(f"gen_mc_tables: wrote {out}")
    return 0


if __name__ == "__main__":
    sys.exit(main(sys.argv))
