"""Generator of csrc/gen_mf60.cuh: the product of one layout-60 sphere pair block with the
source's 60 coefficients, for a target outside the source, without forming the block.

Outside a sphere the potentials of a polynomial eigenstrain are finite sums of derivatives of
r and 1/r (V = 4 pi / 3, unit radius; phi: density / r, psi: density * r)
    1:       phi = V / r                                  psi = V (r + 1 / (5 r))
    x_p:     phi = -V/5 d_p (1/r)                         psi = -V/5 d_p r - V/35 d_p (1/r)
    x_p x_q: phi = V/5 delta_pq / r + V/35 d_pq (1/r)     psi = V/5 delta_pq r + V/35 delta_pq / r
                                                                + V/35 d_pq r + V/315 d_pq (1/r)
and the strains and their derivatives are the D tensors of the reference
(integratorElastic3DHelper.cpp:2394-2554) built from them.  In a frame whose z axis is the
offset x the block couples only components of equal angular order m about z, and each of its
entries is a sum of two or three powers 1/r^k: 520 entries instead of 3,600.  So the product is
    rotate the coefficients into the frame (566 multiply-adds),
    the sparse block (about 520),
    rotate the strains and their derivatives back (about 580),
against 3,600 multiply-adds on top of the ~25,000 operations that form the dense block.

Components.  A symmetric tensor is handled as six numbers (tr, zz, c2, s2, c1, s1): on the way
in tr = E_ii, zz = z.E.z, c2 = x.E.x - y.E.y, s2 = 2 x.E.y, c1 = 2 x.E.z, s1 = 2 y.E.z, i.e.
G_a : E with the matrices G_a = I, zz, xx - yy, xy + yx, xz + zx, yz + zy; on the way out
e = sum_a w_a G_a with the same matrices.  (c1, s1), (c2, s2) and a vector's (x, y) are real and
imaginary parts of components of order m = 1, 2, 1; products of them are combined into
components of definite order before and after the sparse block.
"""
from __future__ import annotations

import functools
from fractions import Fraction as Fr

SYM = [(i, j) for i in range(3) for j in range(i, 3)]
TR, ZZ, C2, S2, C1, S1 = range(6)
GEN = [((0, 0, 1), (1, 1, 1), (2, 2, 1)), ((2, 2, 1),), ((0, 0, 1), (1, 1, -1)), ((0, 1, 1), (1, 0, 1)),
       ((0, 2, 1), (2, 0, 1)), ((1, 2, 1), (2, 1, 1))]


@functools.lru_cache(None)
def _d_pow(s: int, alpha: tuple) -> int:
    """The derivative alpha of r^s at (0, 0, 1) (at (0, 0, r) it is this times r^(s - |alpha|))."""
    if sum(alpha) == 0:
        return 1
    i = next(t for t in range(3) if alpha[t])
    b = alpha[:i] + (alpha[i] - 1,) + alpha[i + 1:]
    v = (1 if i == 2 else 0) * _d_pow(s - 2, b)
    if b[i]:
        v += b[i] * _d_pow(s - 2, b[:i] + (b[i] - 1,) + b[i + 1:])
    return s * v


def _pot(psi: bool, mom: tuple) -> list:
    """[(power of r, derivative indices, factor / V)]."""
    if len(mom) == 0:
        return [(1, (), Fr(1)), (-1, (), Fr(1, 5))] if psi else [(-1, (), Fr(1))]
    if len(mom) == 1:
        return [(1, mom, Fr(-1, 5)), (-1, mom, Fr(-1, 35))] if psi else [(-1, mom, Fr(-1, 5))]
    out = [(1, mom, Fr(1, 35)), (-1, mom, Fr(1, 315))] if psi else [(-1, mom, Fr(1, 35))]
    if mom[0] == mom[1]:
        out += [(1, (), Fr(1, 5)), (-1, (), Fr(1, 35))] if psi else [(-1, (), Fr(1, 5))]
    return out


def _alpha(idx) -> tuple:
    return (idx.count(0), idx.count(1), idx.count(2))


def _d(i, j, k, l, mom, der) -> dict:
    """D_ijkl / V without 1 / (8 pi (1 - nu)) at (0, 0, r): {(k, nu power): factor of 1/r^k nu^p}."""
    out: dict = {}

    def add(psi, idx, c0, c1):
        for s, m, f in _pot(psi, mom):
            a = _alpha(idx + m + der)
            v = f * _d_pow(s, a)
            if v:
                key = sum(a) - s
                out[(key, 0)] = out.get((key, 0), Fr(0)) + c0 * v
                out[(key, 1)] = out.get((key, 1), Fr(0)) + c1 * v

    add(True, (k, l, i, j), 1, 0)
    if k == l:
        add(False, (i, j), 0, -2)
    for hit, idx in ((i == l, (k, j)), (j == l, (k, i)), (i == k, (l, j)), (j == k, (l, i))):
        if hit:
            add(False, idx, -1, 1)
    return out


# ---- components: every source / target component as a combination of tensor entries
def _pair(a, b, name):
    """Real and imaginary combinations of two (re, im) component pairs: sum and difference orders."""
    (ar, ai), (br, bi) = a, b
    return [(f"{name}dr", {(ar, br): 1, (ai, bi): 1}), (f"{name}di", {(ai, br): 1, (ar, bi): -1}),
            (f"{name}sr", {(ar, br): 1, (ai, bi): -1}), (f"{name}si", {(ar, bi): 1, (ai, br): 1})]


def components():
    """[(order, name, {index tuple of the rotated arrays: factor})] of the 60 components, grouped so that the
    sparse block is as sparse as the angular orders allow."""
    out = [(0, f"e{a}", {(a,): 1}) for a in range(6)]
    for a in (TR, ZZ):
        out += [(1, f"f{a}{p}", {(a, p): 1}) for p in range(3)]
    for a in (C2, S2, C1, S1):
        out.append((1, f"f{a}2", {(a, 2): 1}))
    for nm, pr in (("f2", (C2, S2)), ("f1", (C1, S1))):
        out += [(1, n, c) for n, c in _pair(pr, (0, 1), nm)]
    for a in (TR, ZZ):
        out += [(2, f"g{a}{b}", {(a, b): 1}) for b in range(6)]
    for a in (C2, S2, C1, S1):
        out += [(2, f"g{a}{b}", {(a, b): 1}) for b in (TR, ZZ)]
    for n1, p1 in (("2", (C2, S2)), ("1", (C1, S1))):
        for n2, p2 in (("2", (C2, S2)), ("1", (C1, S1))):
            out += [(2, n, c) for n, c in _pair(p1, p2, f"g{n1}_{n2}")]
    assert len(out) == 60
    return out


def _entries(order, comb):
    """Expand a component over Cartesian index tuples (i, j[, p][, q]): {indices: factor}."""
    out: dict = {}
    for idx, f in comb.items():
        for i, j, s in GEN[idx[0]]:
            if order == 0:
                rest = [((), 1)]
            elif order == 1:
                rest = [((idx[1],), 1)]
            else:
                rest = [((p, q), t) for p, q, t in GEN[idx[1]]]
            for m, t in rest:
                key = (i, j) + m
                out[key] = out.get(key, Fr(0)) + f * s * t
    return out


def _solve(basis, vec):
    """Coordinates of the rows `vec` in `basis` (exact Gaussian elimination): list of dicts."""
    n = len(basis)
    keys = sorted({k for b in basis for k in b})
    m = [[b.get(k, Fr(0)) for b in basis] + [v.get(k, {}) for v in vec] for k in keys]
    # columns: n basis coefficients, then dict-valued right-hand sides
    row = 0
    piv = []
    for c in range(n):
        p = next(r for r in range(row, len(m)) if m[r][c] != 0)
        m[row], m[p] = m[p], m[row]
        inv = 1 / m[row][c]
        m[row] = [v * inv for v in m[row][:n]] + [{k: x * inv for k, x in v.items()} for v in m[row][n:]]
        for r in range(len(m)):
            if r != row and m[r][c] != 0:
                f = m[r][c]
                m[r] = [x - f * y for x, y in zip(m[r][:n], m[row][:n])] + [
                    {k: x.get(k, Fr(0)) - f * y.get(k, Fr(0)) for k in set(x) | set(y)} for x, y in zip(m[r][n:], m[row][n:])]
        piv.append(row)
        row += 1
    for r in range(row, len(m)):
        assert all(not any(v.values()) for v in m[r][n:])
    return [[m[piv[c]][n + t] for c in range(n)] for t in range(len(vec))]


@functools.lru_cache(None)
def sparse_block():
    """{(target component, source component): {(k, nu power): factor}} of w = S v, where v are the source
    components (contractions with the coefficients) and the strain derivatives are sum_t w_t (component t's tensor)."""
    comps = components()
    out = {}
    for ro in range(3):
        rows = [(t, c) for t, c in enumerate(comps) if c[0] == ro]
        basis = [_entries(ro, c[2]) for _, c in rows]
        for co in range(3):
            cols = [(u, c) for u, c in enumerate(comps) if c[0] == co]
            cart = sorted({k for _, c in cols for k in _entries(co, c[2])})
            # the dense block over full Cartesian indices: strain (i, j, der) from coefficient (k, l, mom)
            rkeys = sorted({k for b in basis for k in b})
            # source: E = sum over Cartesian entries; v_u = sum E * entries_u.  The dual basis expresses E by v, so the
            # column of component u is the field of the tensor dual to it: tensors T_u = entries_u / |entries_u|^2
            # (the components are mutually orthogonal except (tr, zz) pairs, handled by the exact solve below)
            ents = [_entries(co, c[2]) for _, c in cols]
            gram = [[sum(a.get(k, Fr(0)) * b.get(k, Fr(0)) for k in cart) for b in ents] for a in ents]
            n = len(ents)
            inv = [[Fr(int(r == c)) for c in range(n)] for r in range(n)]
            g = [r[:] for r in gram]
            for c in range(n):
                p = next(r for r in range(c, n) if g[r][c] != 0)
                g[c], g[p], inv[c], inv[p] = g[p], g[c], inv[p], inv[c]
                f = 1 / g[c][c]
                g[c], inv[c] = [v * f for v in g[c]], [v * f for v in inv[c]]
                for r in range(n):
                    if r != c and g[r][c] != 0:
                        f = g[r][c]
                        g[r] = [x - f * y for x, y in zip(g[r], g[c])]
                        inv[r] = [x - f * y for x, y in zip(inv[r], inv[c])]
            dual = []
            for u in range(n):
                t: dict = {}
                for w in range(n):
                    if inv[u][w]:
                        for k, v in ents[w].items():
                            t[k] = t.get(k, Fr(0)) + inv[u][w] * v
                dual.append({k: v for k, v in t.items() if v})
            fields = []
            for t in dual:
                fld: dict = {}
                for rk in rkeys:
                    acc: dict = {}
                    for ck, v in t.items():
                        for kk, x in _d(rk[0], rk[1], ck[0], ck[1], ck[2:], rk[2:]).items():
                            acc[kk] = acc.get(kk, Fr(0)) + v * x
                    acc = {k: v for k, v in acc.items() if v}
                    if acc:
                        fld[rk] = acc
                fields.append(fld)
            for (u, _), coords in zip(cols, _solve(basis, fields)):
                for (t, _), d in zip(rows, coords):
                    d = {k: v for k, v in d.items() if v}
                    if d:
                        out[(t, u)] = d
    return out


def _lit(v: Fr) -> str:
    return f"R({float(v)!r})"


def generate_source() -> str:
    comps = components()
    blk = sparse_block()
    src_off = lambda order, idx: {0: "A0[%d]", 1: "A1[%d][%d]", 2: "A2[%d][%d]"}[order] % idx
    o = []
    o.append("// GENERATED by ibemproject_gb300/codegen_mf60.py -- do not edit by hand.")
    o.append("// Sparse part of the layout-60 pair product in the frame of the offset: source components A0, A1,")
    o.append("// A2 (order 0, 1, 2) to target components W (order RO), %d nonzero entries in all; q[n] = r^-(n + 3)," % len(blk))
    o.append("// nu the matrix's Poisson ratio; without the factor V / (8 pi (1 - nu)).")
    o.append("#pragma once")
    o.append("")
    for ro in range(3):
        dims = {0: "[6]", 1: "[6][3]", 2: "[6][6]"}
        o.append("template <class R>")
        o.append(f"IBEM_HD IBEM_INLINE void mf60_sparse_r{ro}(const R (&A0)[6], const R (&A1)[6][3], const R (&A2)[6][6],")
        o.append(f"                                       const R (&q)[7], R nu, R (&W){dims[ro]}) {{")
        rows = [(t, c) for t, c in enumerate(comps) if c[0] == ro]
        # coefficient polynomials up to a scalar
        polys: dict = {}
        scaled: dict = {}
        need: dict = {}
        for t, _ in rows:
            for u in range(60):
                d = blk.get((t, u))
                if not d:
                    continue
                ks = sorted(d)
                lead = d[ks[0]]
                canon = tuple((k, d[k] / lead) for k in ks)
                need[(t, u)] = (canon, lead)
        # source combinations used
        used = sorted({u for (_, u) in need})
        for u in used:
            co, nm, comb = comps[u]
            if len(comb) > 1:
                items = list(comb.items())
                expr = src_off(co, items[0][0])
                for idx, f in items[1:]:
                    expr += (" + " if f > 0 else " - ") + src_off(co, idx)
                o.append(f"  const R {nm} = {expr};")
        val = lambda u: comps[u][1] if len(comps[u][2]) > 1 else src_off(comps[u][0], next(iter(comps[u][2])))
        npoly = 0
        for canon, lead in need.values():
            if canon not in polys:
                by_k: dict = {}
                for (k, p), f in canon:
                    by_k.setdefault(k, {})[p] = f
                terms = []
                for k in sorted(by_k):
                    f0, f1 = by_k[k].get(0, Fr(0)), by_k[k].get(1, Fr(0))
                    qn = f"q[{k - 3}]"
                    if f1 == 0:
                        terms.append(qn if f0 == 1 else f"{_lit(f0)} * {qn}")
                    elif f0 == 0:
                        terms.append(f"{_lit(f1)} * nu * {qn}")
                    else:
                        terms.append(f"({_lit(f0)} + {_lit(f1)} * nu) * {qn}")
                polys[canon] = f"c{npoly}"
                npoly += 1
                o.append(f"  const R {polys[canon]} = {' + '.join(terms)};")
        nsc = 0
        for canon, lead in need.values():
            key = (canon, abs(lead))
            if key not in scaled:
                if abs(lead) == 1:
                    scaled[key] = polys[canon]
                else:
                    scaled[key] = f"d{nsc}"
                    nsc += 1
                    o.append(f"  const R {scaled[key]} = {_lit(abs(lead))} * {polys[canon]};")
        for t, c in rows:
            expr = ""
            for u in range(60):
                if (t, u) in need:
                    canon, lead = need[(t, u)]
                    term = f"{scaled[(canon, abs(lead))]} * {val(u)}"
                    expr += (term if not expr and lead > 0 else ("-" + term if not expr else (" + " if lead > 0 else " - ") + term))
            o.append(f"  const R w_{c[1]} = {expr or 'R(0)'};")
        # target arrays from the components
        tgt: dict = {}
        for t, c in rows:
            for idx, f in c[2].items():
                tgt.setdefault(idx, []).append((f, f"w_{c[1]}"))
        for idx in sorted(tgt):
            expr = ""
            for f, nm in tgt[idx]:
                expr += (nm if not expr and f > 0 else ("-" + nm if not expr else (" + " if f > 0 else " - ") + nm))
            o.append("  W" + "".join(f"[{i}]" for i in idx) + f" = {expr};")
        o.append("}")
        o.append("")
    return "\n".join(o)


if __name__ == "__main__":
    src = generate_source()
    blk = sparse_block()
    print(len(blk), "entries", len(src.splitlines()), "lines")
    import re
    print({k: len(re.findall(k, src)) for k in (r"const R c\d+", r"const R d\d+", r"const R w_")})
