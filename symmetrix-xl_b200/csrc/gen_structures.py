"""Emits csrc/generated/structures.h: the coupling structure of each supported model
shape as X-macro lists, so that the CUDA kernels expand into straight-line code with
every row, coupling term and monomial index a compile-time constant.

Run from the repository root:  python symmetrix-xl_b200/csrc/gen_structures.py
The tables come from symmetrix-xl_b200/structure.py (first-principles derivation) plus
the extra zero-weight monomials modelgen.model_tables adds for the (3,1) shape.
"""
from __future__ import annotations

import importlib.util
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[2]
PKG = ROOT / "symmetrix-xl_b200"


def _load_pkg():
    spec = importlib.util.spec_from_file_location(
        "symmetrix_xl_b200", PKG / "__init__.py", submodule_search_locations=[str(PKG)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["symmetrix_xl_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# (name, edge l_max, hidden L_max, number of path sets of the split layer-1 kernels, optional explicit sets)
# S2: set 0 = all paths with source l = 0 or 1 (88 rows, 4 source components), sets 1 and 2 share the
# source l = 2 paths (80 and 75 rows, 5 source components each)
SHAPES = [("S0", 3, 0, 1, None), ("S1", 3, 1, 1, None),
          ("S2", 3, 2, 3, [[0, 3, 8, 13, 1, 4, 5, 9, 10, 14], [7, 2, 6, 11], [16, 12, 15]])]


def reverse_path_lines(p, q, l, l1, l2, base, fed):
    """Straight-line gradient code of one path for one (edge, channel): q = index of the path's radial
    function in R[] / dR[], base = first row adjoint of the path in adj[].  With w_a = sum_b h_b adj_ab and
    s_b = sum_a y_a adj_ab the path contributes
      ang_a += R w_a   (angular part of the force),   hadj_b += R s_b   (source adjoint),
      radial += dR * sum_a y_a w_a,   and   sum_a y_a w_a = sum_b h_b s_b.
    The radial sum runs over the shorter index set, and R is folded into that set's vector first, so
    that the other contraction accumulates straight into its target.  Rows outside `fed` have no coupling
    term (their adjoint is zero: 12 of 88 for hidden 0e+1o) and are left out."""
    n1, n2 = 2 * l1 + 1, 2 * l2 + 1
    out = [f"    {{ /* path {p}: edge l={l1}, source l={l2} -> l={l} */"]
    out.append("      float yw = 0.0f;")

    def rows(pairs):
        return [(a, b, base + a * n2 + b) for a, b in pairs if base + a * n2 + b in fed]

    def nested(terms):
        expr = f"{terms[0][0]} * {terms[0][1]}"
        for x, adj in terms[1:]:
            expr = f"fmaf({x}, {adj}, {expr})"
        return expr

    if n2 < n1:
        for b in range(n2):
            out.append(f"      const float rh{b} = R[{q}] * h[{l2 * l2 + b}];")
        for a, b, row in rows((a, b) for a in range(n1) for b in range(n2)):
            out.append(f"      ang[{l1 * l1 + a}] = fmaf(rh{b}, adj[{row}], ang[{l1 * l1 + a}]);")
        for b in range(n2):
            terms = [(f"y[{l1 * l1 + a}]", f"adj[{row}]") for a, _, row in rows((a, b) for a in range(n1))]
            if terms:
                out.append(f"      {{ const float s_ = {nested(terms)};")
                out.append(f"        hadj[{l2 * l2 + b}] = fmaf(R[{q}], s_, hadj[{l2 * l2 + b}]); yw = fmaf(h[{l2 * l2 + b}], s_, yw); }}")
    else:
        for a in range(n1):
            out.append(f"      const float ry{a} = R[{q}] * y[{l1 * l1 + a}];")
        for a in range(n1):
            terms = [(f"h[{l2 * l2 + b}]", f"adj[{row}]") for _, b, row in rows((a, b) for b in range(n2))]
            if terms:
                out.append(f"      {{ const float w = {nested(terms)};")
                out.append(f"        ang[{l1 * l1 + a}] = fmaf(R[{q}], w, ang[{l1 * l1 + a}]); yw = fmaf(y[{l1 * l1 + a}], w, yw); }}")
        for a, b, row in rows((a, b) for b in range(n2) for a in range(n1)):
            out.append(f"      hadj[{l2 * l2 + b}] = fmaf(ry{a}, adj[{row}], hadj[{l2 * l2 + b}]);")
    out.append(f"      radial = fmaf(dR[{q}], yw, radial);")
    out.append("    }")
    return out


def contraction_lines(terms):
    """Straight-line bodies of a symmetric contraction, terms = [(out, term, monomial)], on channel pairs: W(t) weight of term
    t, x[] inputs, o[] outputs (start at zero), adj[] output adjoints, g[] input adjoints (start at zero).

    The monomials of degree 2 and 3 are grouped by their first two factors a, b, so that the products a b and the sums over
    the third factor are formed once per group:
      forward   o[out] += (x_a x_b) (sum_c w x_c + w_ab)                          one operation per term and one per group
      reverse   s = sum_out w adj;  g_c += s x_a x_b;  v = sum_c s x_c + s_ab;  g_a += v x_b;  g_b += v x_a
                                                                                  three per term, three per group
    against three and seven operations for every term on its own."""
    fwd, rev, pairs = [], [], {}
    for out, t, mono in terms:
        if len(mono) == 1:
            fwd.append(f"      o[{out}] = f2_fma(W({t}), x[{mono[0]}], o[{out}]);")
            rev.append(f"      g[{mono[0]}] = f2_fma(W({t}), adj[{out}], g[{mono[0]}]);")
        else:
            third = mono[2] if len(mono) == 3 else None
            pairs.setdefault((mono[0], mono[1]), {}).setdefault(third, []).append((out, t))
    for (a, b), group in sorted(pairs.items()):
        fwd_group, rev_group = [], []     # a group is one line of the header
        thirds = sorted(group, key=lambda c: (c is not None, c))
        fwd_group.append(f"      {{ const unsigned long long p = f2_mul(x[{a}], x[{b}]);")
        for out in sorted({o for c in thirds for o, _ in group[c]}):
            expr = None
            for c in thirds:
                for o, t in group[c]:
                    if o == out:
                        if c is None:
                            expr = f"W({t})" if expr is None else f"f2_add({expr}, W({t}))"
                        else:
                            expr = f"f2_mul(W({t}), x[{c}])" if expr is None else f"f2_fma(W({t}), x[{c}], {expr})"
            fwd_group.append(f"        o[{out}] = f2_fma(p, {expr}, o[{out}]);")
        fwd_group.append("      }")
        cubic = any(c is not None for c in thirds)
        rev_group.append("      {" + (f" const unsigned long long p = f2_mul(x[{a}], x[{b}]);" if cubic else "") + " unsigned long long v;")
        first = True
        for c in thirds:
            expr = None
            for o, t in group[c]:
                expr = f"f2_mul(W({t}), adj[{o}])" if expr is None else f"f2_fma(W({t}), adj[{o}], {expr})"
            if c is None:
                rev_group.append(f"        v = {expr};")
            else:
                rev_group.append(f"        {{ const unsigned long long s = {expr}; g[{c}] = f2_fma(s, p, g[{c}]); "
                           + (f"v = f2_mul(s, x[{c}]); }}" if first else f"v = f2_fma(s, x[{c}], v); }}"))
            first = False
        rev_group.append(f"        g[{a}] = f2_fma(v, x[{b}], g[{a}]); g[{b}] = f2_fma(v, x[{a}], g[{b}]);")
        rev_group.append("      }")
        fwd.append("      " + " ".join(part.strip() for part in fwd_group))
        rev.append("      " + " ".join(part.strip() for part in rev_group))
    return fwd, rev


ROW_BATCH = 8      # kRowBatch of edge_kernels_pairs.cuh


def reverse_edges_lines(paths, row_begin, fed):
    """Straight-line layer-1 gradient of one edge on channel pairs (edge_kernels_pairs.cuh) and the rows in the order it uses
    them.  Row adjoints come kRowBatch at a time: ROWS(batch) brings the batch into w[], every value of which feeds two
    operations.  Names: h[lm2], hadj[lm2] source features and their adjoint, R, dR radial value and slope of the path at hand
    (RADIAL(p) fetches them), y[], ang[] the harmonics and the angular adjoint of the edge l at hand (f[lm]: of both channels),
    radial.  Per path the same
    contractions as reverse_path_lines; rows that no coupling term feeds (their adjoint is zero: 12 of 88 for hidden 0e+1o, 56
    of 243 for 0e+1o+2e) are left out."""
    out, used, order = [], set(), []

    def put(target, a, b):
        out[-1] += f" {target} = f2_fma({a}, {b}, {target});" if target in used else f" {target} = f2_mul({a}, {b});"
        used.add(target)

    def take(row):
        slot = len(order)
        order.append(row)
        out.append(f"      {f'ROWS({slot // ROW_BATCH}) ' if slot % ROW_BATCH == 0 else ''}{{ const f2 w = rows[{slot % ROW_BATCH}];")

    for l1 in sorted({path[1] for path in paths}):
        n1 = 2 * l1 + 1
        out.append(f"    {{ f2 y[{n1}]{f', ang[{n1}]' if l1 else ''}; load_pair_harmonics<{l1}>(yrow, y);")
        used -= {f"ang[{a}]" for a in range(16)}
        for p, (l, _, l2) in [(p, path) for p, path in enumerate(paths) if path[1] == l1]:
            n2 = 2 * l2 + 1
            out.append(f"    {{ /* path {p}: edge l={l1}, source l={l2} -> l={l} */ RADIAL({p}) f2 yw, t[{n2}], v[{n2}];")
            used -= {"yw"} | {f"{k}[{q}]" for k in "tv" for q in range(16)}
            if n2 < n1:
                for b in range(n2):
                    out.append("     ")
                    put(f"t[{b}]", "R", f"h[{l2 * l2 + b}]")
                for a in range(n1):
                    for b in range(n2):
                        if row_begin[p] + a * n2 + b not in fed:
                            continue
                        take(row_begin[p] + a * n2 + b)
                        put(f"ang[{a}]", f"t[{b}]", "w")
                        put(f"v[{b}]", f"y[{a}]", "w")
                        out[-1] += " }"
                for b in range(n2):
                    out.append("     ")
                    put(f"hadj[{l2 * l2 + b}]", "R", f"v[{b}]")
                    put("yw", f"h[{l2 * l2 + b}]", f"v[{b}]")
            else:
                for a in range(n1):
                    row = row_begin[p] + a * n2
                    if not fed.intersection(range(row, row + n2)):
                        continue
                    out.append(f"      t[0] = f2_mul(R, y[{a}]);")
                    used -= {"v[0]"}
                    for b in range(n2):
                        if row + b not in fed:
                            continue
                        take(row + b)
                        put("v[0]", f"h[{l2 * l2 + b}]", "w")
                        put(f"hadj[{l2 * l2 + b}]", "t[0]", "w")
                        out[-1] += " }"
                    out.append("     ")
                    if l1:
                        put(f"ang[{a}]", "R", "v[0]")
                    put("yw", f"y[{a}]", "v[0]")
            out.append("     ")
            put("radial", "dR", "yw")
            out.append("    }")
        if l1:
            out.append("     " + "".join(f" f[{l1 * l1 + a}] = f2_sum(ang[{a}]);" for a in range(n1)))
        out.append("    }")
    return out, order


def adjoint_rows_lines(order, term_row, term_lme):
    """The row adjoints in that order, kRowBatch at a time: TERM(slot, term, lme) / TERM_ADD for a row's first / further coupling
    terms, STORE(batch) hands a full batch (the last one padded with zeros) over."""
    out = []
    for slot, row in enumerate(order + [None] * (-len(order) % ROW_BATCH)):
        terms = [(t, lme) for t, (r, lme) in enumerate(zip(term_row, term_lme)) if r == row]
        line = "    " + (" ".join(f"TERM{'_ADD' if n else ''}({slot % ROW_BATCH}, {t}, {lme})" for n, (t, lme) in enumerate(terms))
                         if terms else f"v[{slot % ROW_BATCH}] = 0ull;")
        if slot % ROW_BATCH == ROW_BATCH - 1:
            line += f" STORE({slot // ROW_BATCH})"
        out.append(line)
    return out


def emit_shape(name, l_max, L_max, tables, groups=1, by_edge_l=None):
    out = []
    paths = list(zip(tables["Phi1_l"], tables["Phi1_l1"], tables["Phi1_l2"]))
    num_lm, num_LM = (l_max + 1) ** 2, (L_max + 1) ** 2
    rows = []
    row_begin = []
    for p, (l, l1, l2) in enumerate(paths):
        row_begin.append(len(rows))
        for lm1 in range(l1 * l1, (l1 + 1) ** 2):
            for lm2 in range(l2 * l2, (l2 + 1) ** 2):
                rows.append((p, lm1, lm2))
    out.append(f"// ---- shape {name}: edge l_max={l_max}, hidden L_max={L_max}")
    out.append(f"#define SXB_{name}_LMAX {l_max}")
    out.append(f"#define SXB_{name}_HIDDEN_LMAX {L_max}")
    out.append(f"#define SXB_{name}_NUM_LM {num_lm}")
    out.append(f"#define SXB_{name}_NUM_HIDDEN {num_LM}")
    out.append(f"#define SXB_{name}_NUM_PATHS {len(paths)}")
    out.append(f"#define SXB_{name}_NUM_ROWS {len(rows)}")
    out.append(f"#define SXB_{name}_NUM_LME {tables['num_lme']}")
    out.append(f"#define SXB_{name}_NUM_TERMS {len(tables['Phi1_lme'])}")
    out.append(f"// X(path, l_out, l_edge, l_source, first_row)")
    out.append(f"#define SXB_{name}_PATHS(X) \\")
    out.append(" \\\n".join(f"    X({p}, {l}, {l1}, {l2}, {row_begin[p]})" for p, (l, l1, l2) in enumerate(paths)))
    out.append(f"// X(row, path, lm_edge, lm_source)")
    out.append(f"#define SXB_{name}_ROWS(X) \\")
    out.append(" \\\n".join(f"    X({r}, {p}, {lm1}, {lm2})" for r, (p, lm1, lm2) in enumerate(rows)))
    out.append(f"// X(term, row, lme): coefficient values live in constant memory, indexed by term")
    out.append(f"#define SXB_{name}_TERMS(X) \\")
    out.append(" \\\n".join(f"    X({t}, {row}, {lme})" for t, (row, lme) in
                            enumerate(zip(tables["Phi1_lelm1lm2"], tables["Phi1_lme"]))))
    out.append(f"// this library's own derivation of the coupling coefficients, by term (a model file carries its own)")
    out.append(f"#define SXB_{name}_DEFAULT_CG {{" + ", ".join(f"{float(v)!r}f" for v in tables["Phi1_clebsch_gordan"]) + "}")
    # symmetric contraction: weights laid out [type][term][channel], term = offset(LM) + index
    offset = 0
    lines1, lines2, lines3 = [], [], []
    offs = []
    for LM in range(num_LM):
        mons = tables["M0_monomials"][str(LM)]
        offs.append(offset)
        for t, mono in enumerate(mons):
            if len(mono) == 1:
                lines1.append(f"    X1({LM}, {offset + t}, {mono[0]})")
            elif len(mono) == 2:
                lines2.append(f"    X2({LM}, {offset + t}, {mono[0]}, {mono[1]})")
            else:
                lines3.append(f"    X3({LM}, {offset + t}, {mono[0]}, {mono[1]}, {mono[2]})")
        offset += len(mons)
    out.append(f"#define SXB_{name}_M0_NUM_TERMS {offset}")
    out.append(f"#define SXB_{name}_M0_OFFSETS {{{', '.join(map(str, offs + [offset]))}}}")
    out.append(f"// X1(out, term, a)  X2(out, term, a, b)  X3(out, term, a, b, c)")
    out.append(f"#define SXB_{name}_M0_TERMS(X1, X2, X3) \\")
    out.append(" \\\n".join(lines1 + lines2 + lines3))
    m1 = tables["M1_monomials"]
    out.append(f"#define SXB_{name}_M1_NUM_TERMS {len(m1)}")
    l1_, l2_, l3_ = [], [], []
    for t, mono in enumerate(m1):
        if len(mono) == 1:
            l1_.append(f"    X1(0, {t}, {mono[0]})")
        elif len(mono) == 2:
            l2_.append(f"    X2(0, {t}, {mono[0]}, {mono[1]})")
        else:
            l3_.append(f"    X3(0, {t}, {mono[0]}, {mono[1]}, {mono[2]})")
    out.append(f"#define SXB_{name}_M1_TERMS(X1, X2, X3) \\")
    out.append(" \\\n".join(l1_ + l2_ + l3_))
    m0 = [(LM, offs[LM] + t, mono) for LM in range(num_LM) for t, mono in enumerate(tables["M0_monomials"][str(LM)])]
    for which, terms in (("M0", m0), ("M1", [(0, t, mono) for t, mono in enumerate(m1)])):
        fwd, rev = contraction_lines(terms)
        out.append(f"#define SXB_{name}_{which}_FORWARD_BODY \\")
        out.append(" \\\n".join(fwd))
        out.append(f"#define SXB_{name}_{which}_REVERSE_BODY \\")
        out.append(" \\\n".join(rev))
    # straight-line bodies of the layer-1 edge kernels (one channel per thread):
    #   R[p], dR[p]: radial value / derivative of path p;  y[lm]: edge harmonics;
    #   h[lm2]: source features;  acc[row] / adj[row]: receiver row sums / row adjoints
    fwd, rev = [], []
    for p, (l, l1, l2) in enumerate(paths):
        n1, n2 = 2 * l1 + 1, 2 * l2 + 1
        fwd.append(f"    {{ /* path {p}: edge l={l1}, source l={l2} -> l={l} */")
        for b in range(n2):
            fwd.append(f"      const float t{b} = R[{p}] * h[{l2 * l2 + b}];")
        for a in range(n1):
            for b in range(n2):
                row = row_begin[p] + a * n2 + b
                fwd.append(f"      acc[{row}] = fmaf(t{b}, y[{l1 * l1 + a}], acc[{row}]);")
        fwd.append("    }")
        rev.extend(reverse_path_lines(p, p, l, l1, l2, row_begin[p], set(tables["Phi1_lelm1lm2"])))
    if groups == 1:      # shapes with path sets have no kernel that holds all rows in registers
        out.append(f"#define SXB_{name}_L1_FORWARD_BODY \\")
        out.append(" \\\n".join(fwd))
        out.append(f"#define SXB_{name}_L1_REVERSE_BODY \\")
        out.append(" \\\n".join(rev))
    if L_max > 0:
        body, order = reverse_edges_lines(paths, row_begin, set(tables["Phi1_lelm1lm2"]))
        out.append(f"#define SXB_{name}_ROW_BATCHES {(len(order) + ROW_BATCH - 1) // ROW_BATCH}")
        out.append(f"#define SXB_{name}_L1_REVERSE_EDGE_BODY \\")
        out.append(" \\\n".join(body))
        out.append(f"#define SXB_{name}_L1_ADJOINT_ROWS \\")
        out.append(" \\\n".join(adjoint_rows_lines(order, tables["Phi1_lelm1lm2"], tables["Phi1_lme"])))
    if groups > 1:
        out.extend(emit_path_groups(name, paths, row_begin, tables, groups, by_edge_l))
    out.append("")
    return "\n".join(out)


def emit_path_groups(name, paths, row_begin, tables, groups, by_edge_l=None):
    """Splits the paths of a shape into `groups` sets with balanced row counts and emits, per set,
    the same straight-line bodies with rows, paths and outputs renumbered inside the set.  Every
    output component (lme) is fed by exactly one path, so the sets write disjoint outputs; a kernel
    instance that handles one set needs only that set's row accumulators in registers."""
    sizes = [(2 * l1 + 1) * (2 * l2 + 1) for (_, l1, l2) in paths]
    members = [[] for _ in range(groups)]
    load = [0] * groups
    if by_edge_l is not None:
        # explicit sets (lists of path indices), chosen so that a set touches few source components:
        # a set loads and atomically updates only the source components of its own paths
        assert sorted(p for group in by_edge_l for p in group) == list(range(len(paths)))
        members = [list(group) for group in by_edge_l]
    else:
        for p in sorted(range(len(paths)), key=lambda q: -sizes[q]):      # largest first, to the lightest set
            g = min(range(groups), key=lambda q: load[q])
            members[g].append(p)
            load[g] += sizes[p]
    row_path = []
    for p, n in enumerate(sizes):
        row_path += [p] * n
    lme_path = {}
    for row, lme in zip(tables["Phi1_lelm1lm2"], tables["Phi1_lme"]):
        assert lme_path.setdefault(lme, row_path[row]) == row_path[row]
    out = [f"#define SXB_{name}_NUM_GROUPS {groups}"]
    for g, plist in enumerate(members):
        plist = sorted(plist)
        local_row, rows_g = {}, 0
        for p in plist:
            for r in range(sizes[p]):
                local_row[row_begin[p] + r] = rows_g
                rows_g += 1
        lmes = sorted(lme for lme, p in lme_path.items() if p in plist)
        local_lme = {lme: i for i, lme in enumerate(lmes)}
        hmask = 0
        for p in plist:
            l2 = paths[p][2]
            for b in range(l2 * l2, (l2 + 1) ** 2):
                hmask |= 1 << b
        pre = f"SXB_{name}_G{g}"
        out.append(f"#define {pre}_NUM_PATHS {len(plist)}")
        out.append(f"#define {pre}_NUM_ROWS {rows_g}")
        out.append(f"#define {pre}_NUM_LME {len(lmes)}")
        out.append(f"#define {pre}_PATH_LIST {{{', '.join(map(str, plist))}}}")
        out.append(f"#define {pre}_LME_LIST {{{', '.join(map(str, lmes))}}}")
        out.append(f"#define {pre}_SOURCE_MASK {hmask}u   // source components lm2 the set touches")
        out.append(f"// X(term, row inside the set, output inside the set)")
        out.append(f"#define {pre}_TERMS(X) \\")
        out.append(" \\\n".join(f"    X({t}, {local_row[row]}, {local_lme[lme]})" for t, (row, lme) in
                                enumerate(zip(tables["Phi1_lelm1lm2"], tables["Phi1_lme"])) if row in local_row))
        fwd = []
        for q, p in enumerate(plist):
            l, l1, l2 = paths[p]
            n1, n2 = 2 * l1 + 1, 2 * l2 + 1
            base = local_row[row_begin[p]]
            fwd.append(f"    {{ /* path {p}: edge l={l1}, source l={l2} -> l={l} */")
            for b in range(n2):
                fwd.append(f"      const float t{b} = R[{q}] * h[{l2 * l2 + b}];")
            for a in range(n1):
                for b in range(n2):
                    row = base + a * n2 + b
                    fwd.append(f"      acc[{row}] = fmaf(t{b}, y[{l1 * l1 + a}], acc[{row}]);")
            fwd.append("    }")
        out.append(f"#define {pre}_FORWARD_BODY \\")
        out.append(" \\\n".join(fwd))
    return out


def main():
    pkg = _load_pkg()
    text = ["// Generated by symmetrix-xl_b200/csrc/gen_structures.py -- do not edit.",
            "// Coupling structure of the supported model shapes as X-macro lists.",
            "#pragma once", ""]
    for name, l_max, L_max, groups, by_edge_l in SHAPES:
        tables = pkg.modelgen.model_tables(l_max, L_max)
        text.append(emit_shape(name, l_max, L_max, tables, groups, by_edge_l))
    target = PKG / "csrc" / "generated" / "structures.h"
    target.write_text("\n".join(text))
    print("wrote", target)


if __name__ == "__main__":
    main()
