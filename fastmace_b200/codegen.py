"""Generates the straight-line CUDA bodies of the channelwise tensor product from the coupling tables.

``python -m fastmace_b200.codegen`` writes ``csrc/generated/tp_generated.cuh`` with, for every node l_max
(0, 1, 2) entering the product:

* ``TpShape<LIN>``: number of paths, input components, components of the scattered message;
* ``tp_forward<0>(x, Y, w, acc)``: ``acc[slot] += w[path] * sum_terms coef * x[m_in] * Y[m_edge]``;
* ``tp_backward<LIN, FLIP, NEED_DX>(x, Y, w, wp, g, dY, dr, dx)``: the adjoint of the same expression for one edge and
  one channel given the gradient ``g`` of the receiver's scattered message. ``FLIP`` evaluates the edge in the opposite
  direction (``Y_l -> (-1)^l Y_l``, folded into the coefficients), which is how a receiver-owned walk also produces
  the sender-side gradient of its mirror edge without atomics.

The message layout is K-contiguous for the per-l linear that follows: inside the block of output irrep l the component
index is ``base_l + m * n_seg(l) + seg`` (m the component, seg the path's rank among the paths into l).

All indices are compile-time constants, so ``x``, ``Y``, ``w``, ``acc`` ... live in registers.
"""

from __future__ import annotations

import os

from . import so3

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.join(HERE, "csrc", "generated", "tp_generated.cuh")


def message_slots(paths):
    """slot[(path, m_out)] -> component index of the K-contiguous message layout; also per-l (base, n_seg)."""
    slots, blocks, base = {}, {}, 0
    for l_out in range(so3.LMAX_SH + 1):
        into = so3.paths_into(paths, l_out)
        blocks[l_out] = (base, len(into))
        for seg, p in enumerate(into):
            for m in range(2 * l_out + 1):
                slots[(p, m)] = base + m * len(into) + seg
        base += len(into) * (2 * l_out + 1)
    return slots, blocks


def _lit(value: float) -> str:
    text = f"{float(value):.9g}"
    if "." not in text and "e" not in text:
        text += ".0"
    return text + "f"


def _emit(lin: int) -> str:
    paths = so3.tp_paths(lin)
    slots, blocks = message_slots(paths)
    in_dim = (lin + 1) ** 2
    mid = so3.mid_dim(paths)
    n_terms = sum(len(p["terms"]) for p in paths)
    out = [f"// ---- node l_max = {lin}: {len(paths)} paths, {mid} message components, {n_terms} coupling terms",
           f"template <> struct TpShape<{lin}> {{",
           f"    static constexpr int kPaths = {len(paths)};",
           f"    static constexpr int kInDim = {in_dim};",
           f"    static constexpr int kMidDim = {mid};",
           "};",
           ""]
    if lin == 0:                          # forward (first interaction; later ones: the coupled bodies)
        out += [f"template <> __device__ __forceinline__ void tp_forward<{lin}>(const float (&x)[{in_dim}], "
                f"const float (&Y)[16], const float (&w)[{len(paths)}], float (&acc)[{mid}]) {{"]
        for p, path in enumerate(paths):
            out.append(f"    // path {p}: {path['l_in']} x {path['l_edge']} -> {path['l_out']}")
            by_out: dict[int, list] = {}
            for mi, me, mo, c in path["terms"]:
                by_out.setdefault(mo, []).append((mi, me, c))
            for mo, terms in sorted(by_out.items()):
                expr = " + ".join(f"{_lit(c)} * x[{path['in_off'] + mi}] * Y[{path['edge_off'] + me}]"
                                  for mi, me, c in terms)
                out.append(f"    acc[{slots[(p, mo)]}] = fmaf(w[{p}], {expr}, acc[{slots[(p, mo)]}]);")
        out += ["}", ""]
    # backward
    out += [f"template <bool FLIP, bool NEED_DX> __device__ __forceinline__ void tp_backward_{lin}("
            f"const float (&x)[{in_dim}], const float (&Y)[16], const float (&w)[{len(paths)}], "
            f"const float (&wp)[{len(paths)}], const float (&g)[{mid}], float (&dY)[16], float& dr, "
            f"float (&dx)[{in_dim}]) {{"]
    for p, path in enumerate(paths):
        sign = -1.0 if path["l_edge"] % 2 else 1.0
        out.append(f"    {{  // path {p}: {path['l_in']} x {path['l_edge']} -> {path['l_out']}")
        out.append(f"        constexpr float sg = FLIP ? {_lit(sign)} : 1.0f;")
        by_edge: dict[int, list] = {}
        by_in: dict[int, list] = {}
        for mi, me, mo, c in path["terms"]:
            by_edge.setdefault(me, []).append((mi, mo, c))
            by_in.setdefault(mi, []).append((me, mo, c))
        out.append("        float dw = 0.0f;")
        for me, terms in sorted(by_edge.items()):
            expr = " + ".join(f"{_lit(c)} * x[{path['in_off'] + mi}] * g[{slots[(p, mo)]}]" for mi, mo, c in terms)
            ye = path["edge_off"] + me
            out.append(f"        {{ const float s = sg * ({expr}); dw = fmaf(s, Y[{ye}], dw); "
                       f"dY[{ye}] = fmaf(w[{p}], s, dY[{ye}]); }}")
        out.append(f"        dr = fmaf(wp[{p}], dw, dr);")
        out.append("        if (NEED_DX) {")
        for mi, terms in sorted(by_in.items()):
            expr = " + ".join(f"{_lit(c)} * Y[{path['edge_off'] + me}] * g[{slots[(p, mo)]}]" for me, mo, c in terms)
            xi = path["in_off"] + mi
            out.append(f"            dx[{xi}] = fmaf(w[{p}] * sg, {expr}, dx[{xi}]);")
        out.append("        }")
        out.append("    }")
    out += ["}", ""]
    # per-l blocks of the message layout for the host (base component, segments)
    out.append(f"template <> struct TpBlocks<{lin}> {{")
    out.append("    static constexpr int kBase[4] = {" + ", ".join(str(blocks[l][0]) for l in range(4)) + "};")
    out.append("    static constexpr int kSegs[4] = {" + ", ".join(str(blocks[l][1]) for l in range(4)) + "};")
    out.append("};")
    out.append("")
    return "\n".join(out)


def render() -> str:
    head = ["// GENERATED by fastmace_b200/codegen.py from fastmace_b200/so3.py -- do not edit.",
            "// Channelwise (uvu) tensor product of node irreps 0..LIN with spherical harmonics l <= 3 into 0e+1o+2e+3o;",
            "// coefficients are sqrt(2 l_out + 1) * wigner_3j(l_in, l_edge, l_out).",
            "#pragma once",
            "",
            "namespace fmb {",
            "",
            "template <int LIN> struct TpShape;",
            "template <int LIN> struct TpBlocks;",
            "template <int LIN> __device__ __forceinline__ void tp_forward(const float (&x)[1], const float (&Y)[16], "
            "const float (&w)[4], float (&acc)[16]);",
            ""]
    body = [_emit(lin) for lin in (0, 1, 2)]
    tail = ["}  // namespace fmb", ""]
    return "\n".join(head + body + tail)


def main() -> str:
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    text = render()
    old = open(OUT).read() if os.path.exists(OUT) else None
    if old != text:
        with open(OUT, "w") as handle:
            handle.write(text)
    return OUT




# --------------------------------------------------------------------------------------------- symmetric contraction
SYMCON_OUT = os.path.join(HERE, "csrc", "generated", "symcon_generated.cuh")


def _emit_symcon(l_out_max: int) -> str:
    """Straight-line forward and backward of the contraction polynomial for outputs 0..l_out_max.

    ``cf`` points at this thread's coefficient column: term t is ``cf[t * 128]`` (table order = so3.contraction_keys).
    Products of a degree-2 prefix are shared by the degree-3 monomials that extend it, as in the reference's generated
    kernels (fastmace/kernels/cuda/sc_generated.py:65-107)."""
    keys = so3.contraction_keys(l_out_max)
    n_out = (l_out_max + 1) ** 2
    index = {key: t for t, key in enumerate(keys)}
    by_mono: dict[tuple, list] = {}
    for (m_out, nu, mono), t in index.items():
        by_mono.setdefault(mono, []).append((m_out, t))
    deg1 = sorted(m for m in by_mono if len(m) == 1)
    deg2 = sorted(m for m in by_mono if len(m) == 2)
    deg3 = sorted(m for m in by_mono if len(m) == 3)
    prefixes = sorted({m[:2] for m in deg3} | set(deg2))
    fwd = [f"template <> struct SymconShape<{l_out_max}> {{ static constexpr int kTerms = {len(keys)}; "
           f"static constexpr int kOut = {n_out}; }};",
           f"template <> __device__ __forceinline__ void symcon_forward_body<{l_out_max}>(const float (&x)[16], "
           f"const float* __restrict__ cf, float (&y)[{n_out}]) {{"]

    def consume(mono, expr, lines):
        for m_out, t in sorted(by_mono.get(mono, ())):
            lines.append(f"    y[{m_out}] = fmaf(__ldg(cf + {t * 128}), {expr}, y[{m_out}]);")

    for mono in deg1:
        consume(mono, f"x[{mono[0]}]", fwd)
    for pre in prefixes:
        fwd.append(f"    {{ const float p = x[{pre[0]}] * x[{pre[1]}];")
        consume(pre, "p", fwd)
        for mono in (m for m in deg3 if m[:2] == pre):
            consume(mono, f"(p * x[{mono[2]}])", fwd)
        fwd.append("    }")
    fwd += ["}", ""]
    bwd = [f"template <> __device__ __forceinline__ void symcon_backward_body<{l_out_max}>(const float (&x)[16], "
           f"const float* __restrict__ cf, const float (&g)[{n_out}], float (&dx)[16]) {{"]

    def adjoint(mono):
        return " + ".join(f"__ldg(cf + {t * 128}) * g[{m_out}]" for m_out, t in sorted(by_mono[mono]))

    for mono in deg1:
        bwd.append(f"    dx[{mono[0]}] += {adjoint(mono)};")
    for pre in prefixes:
        i, j = pre
        extended = any(m[:2] == pre for m in deg3)
        bwd.append(f"    {{ {f'const float p = x[{i}] * x[{j}]; ' if extended else ''}float hp = 0.0f;")
        if pre in by_mono:
            bwd.append(f"      hp += {adjoint(pre)};")
        for mono in (m for m in deg3 if m[:2] == pre):
            k = mono[2]
            bwd.append(f"      {{ const float h = {adjoint(mono)}; dx[{k}] = fmaf(h, p, dx[{k}]); hp = fmaf(h, x[{k}], hp); }}")
        bwd.append(f"      dx[{i}] = fmaf(hp, x[{j}], dx[{i}]); dx[{j}] = fmaf(hp, x[{i}], dx[{j}]);")
        bwd.append("    }")
    bwd += ["}", ""]
    return "\n".join(fwd + bwd)


SYMCON_PARTS = (1, 2)


def _emit_symcon_group(l_out_max: int) -> str:
    """The same polynomial for the four atoms of a group at once, two pairs on the packed FP32 pipe: every coefficient is
    loaded once and used four times. ``part`` of ``parts`` evaluates a run of the monomials only (the parts' results are
    added afterwards), so that several warps share a (group, channel block)."""
    keys = so3.contraction_keys(l_out_max)
    n_out = (l_out_max + 1) ** 2
    index = {key: t for t, key in enumerate(keys)}
    by_mono: dict[tuple, list] = {}
    for (m_out, nu, mono), t in index.items():
        by_mono.setdefault(mono, []).append((m_out, t))
    deg1 = sorted(m for m in by_mono if len(m) == 1)
    deg2 = sorted(m for m in by_mono if len(m) == 2)
    deg3 = sorted(m for m in by_mono if len(m) == 3)
    prefixes = sorted({m[:2] for m in deg3} | set(deg2))
    loop = "_Pragma(\"unroll\") for (int r = 0; r < 2; ++r)"

    def weight(t):
        return f"const float2 w = symcon_pair(__ldg(cf + {t * 128}));"

    def fwd_terms(mono, value):
        return [f"      {{ {weight(t)} {loop} y[r][{m_out}] = __ffma2_rn(w, {value}, y[r][{m_out}]); }}"
                for m_out, t in sorted(by_mono.get(mono, ()))]

    def bwd_terms(mono, target):
        return [f"      {{ {weight(t)} {loop} {target}[r] = __ffma2_rn(w, g[r][{m_out}], {target}[r]); }}"
                for m_out, t in sorted(by_mono[mono])]

    zero = "make_float2(0.0f, 0.0f)"
    fwd_blocks, bwd_blocks = [], []                                   # (terms, lines)
    for mono in deg1:
        n = len(by_mono[mono])
        fwd_blocks.append((n, fwd_terms(mono, f"x[r][{mono[0]}]")))
        bwd_blocks.append((n, [f"    {{ float2 h[2]; {loop} h[r] = {zero};", *bwd_terms(mono, "h"),
                               f"      {loop} dx[r][{mono[0]}] = __fadd2_rn(dx[r][{mono[0]}], h[r]); }}"]))
    for pre in prefixes:
        i, j = pre
        longer = [m for m in deg3 if m[:2] == pre]
        n = len(by_mono.get(pre, ())) + sum(len(by_mono[m]) for m in longer)
        lines = [f"    {{ float2 p[2]; {loop} p[r] = __fmul2_rn(x[r][{i}], x[r][{j}]);", *fwd_terms(pre, "p[r]")]
        for mono in longer:
            lines += [f"      {{ float2 q[2]; {loop} q[r] = __fmul2_rn(p[r], x[r][{mono[2]}]);", *fwd_terms(mono, "q[r]"), "      }"]
        fwd_blocks.append((n, lines + ["    }"]))
        lines = [f"    {{ float2 p[2], hp[2]; {loop} {{ p[r] = __fmul2_rn(x[r][{i}], x[r][{j}]); hp[r] = {zero}; }}" if longer
                 else f"    {{ float2 hp[2]; {loop} hp[r] = {zero};"]
        if pre in by_mono:
            lines += bwd_terms(pre, "hp")
        for mono in longer:
            k = mono[2]
            lines += [f"      {{ float2 h[2]; {loop} h[r] = {zero};", *bwd_terms(mono, "h"),
                      f"        {loop} {{ dx[r][{k}] = __ffma2_rn(h[r], p[r], dx[r][{k}]); hp[r] = __ffma2_rn(h[r], x[r][{k}], hp[r]); }} }}"]
        lines += [f"      {loop} {{ dx[r][{i}] = __ffma2_rn(hp[r], x[r][{j}], dx[r][{i}]); "
                  f"dx[r][{j}] = __ffma2_rn(hp[r], x[r][{i}], dx[r][{j}]); }}", "    }"]
        bwd_blocks.append((n, lines))

    def split(blocks, parts):
        total, out, done = sum(n for n, _ in blocks), [[] for _ in range(parts)], 0
        for n, lines in blocks:
            out[min(parts - 1, (2 * done + n) * parts // (2 * total))] += lines
            done += n
        return out

    text = []
    for parts in SYMCON_PARTS:
        for head, blocks in (
                (f"template <> __device__ __forceinline__ void symcon_forward_group<{l_out_max}, {parts}>(int part, const float2 (&x)[2][16], "
                 f"const float* __restrict__ cf, float2 (&y)[2][{n_out}]) {{", fwd_blocks),
                (f"template <> __device__ __forceinline__ void symcon_backward_group<{l_out_max}, {parts}>(int part, const float2 (&x)[2][16], "
                 f"const float* __restrict__ cf, const float2 (&g)[2][{n_out}], float2 (&dx)[2][16]) {{", bwd_blocks)):
            text.append(head)
            for q, lines in enumerate(split(blocks, parts)):
                text += [f"    {'else ' if q else ''}if (part == {q}) {{", *lines, "    }"]
            text += ["}", ""]
    return "\n".join(text)


def render_symcon() -> str:
    head = ["// GENERATED by fastmace_b200/codegen.py from fastmace_b200/so3.py -- do not edit.",
            "// Symmetric contraction (correlation 3) of the 16 message components as a polynomial per (atom, channel):",
            "// y[M] = sum_t coef[species][t][channel] * monomial_t(x), terms in the order of so3.contraction_keys.",
            "#pragma once",
            "",
            "namespace fmb {",
            "",
            "template <int LOUT> struct SymconShape;",
            "template <int LOUT> __device__ __forceinline__ void symcon_forward_body(const float (&x)[16], "
            "const float* __restrict__ cf, float (&y)[(LOUT + 1) * (LOUT + 1)]);",
            "template <int LOUT> __device__ __forceinline__ void symcon_backward_body(const float (&x)[16], "
            "const float* __restrict__ cf, const float (&g)[(LOUT + 1) * (LOUT + 1)], float (&dx)[16]);",
            "__device__ __forceinline__ float2 symcon_pair(float v) { return make_float2(v, v); }",
            "template <int LOUT, int PARTS> __device__ __forceinline__ void symcon_forward_group(int part, const float2 (&x)[2][16], "
            "const float* __restrict__ cf, float2 (&y)[2][(LOUT + 1) * (LOUT + 1)]);",
            "template <int LOUT, int PARTS> __device__ __forceinline__ void symcon_backward_group(int part, const float2 (&x)[2][16], "
            "const float* __restrict__ cf, const float2 (&g)[2][(LOUT + 1) * (LOUT + 1)], float2 (&dx)[2][16]);",
            ""]
    return "\n".join(head + [_emit_symcon(l) for l in (0, 1, 2)] + [_emit_symcon_group(l) for l in (0, 1, 2)] +
                     ["}  // namespace fmb", ""])


def _write(path: str, text: str) -> None:
    os.makedirs(os.path.dirname(path), exist_ok=True)
    old = open(path).read() if os.path.exists(path) else None
    if old != text:
        with open(path, "w") as handle:
            handle.write(text)


# --------------------------------------------------------------------------------------------- coupled bodies
COUPLED_OUT = os.path.join(HERE, "csrc", "generated", "tp_coupled_generated.cuh")


def coupled_layout(paths):
    """Where the couplings of an edge stand: T[path][m_out][m_in] = sum_me coef * Y[me], structural zeros left out. Returns
    ({(path, m_out, m_in): offset}, {offset: [(edge component, coef)]}, floats); the row stride is 4 mod 32 floats so that
    the rows of neighbouring edges start in different banks."""
    offset, sums, at = {}, {}, 0
    for p, path in enumerate(paths):
        for mi, me, mo, c in sorted(path["terms"], key=lambda t: (t[2], t[0], t[1])):
            if (p, mo, mi) not in offset:
                offset[p, mo, mi] = at
                sums[at] = []
                at += 1
            sums[offset[p, mo, mi]].append((path["edge_off"] + me, c))
    stride = -(-at // 4) * 4
    while stride % 32 != 4:
        stride += 4
    return offset, sums, stride


def _emit_coupled(lin: int) -> str:
    """Bodies for two channels per thread (packed FP32, fma.rn.f32x2) that take the harmonics already coupled: what an edge
    needs of them is the small matrix T of every path, the same for all channels."""
    paths = so3.tp_paths(lin)
    slots, _ = message_slots(paths)
    in_dim, mid = (lin + 1) ** 2, so3.mid_dim(paths)
    offset, sums, stride = coupled_layout(paths)
    out = [f"// ---- node l_max = {lin}"]
    # how each coupling is made, for a thread per coupling: c0 Y[at & 15] + c1 Y[at >> 8 & 15], stored at at >> 16
    order = sorted(sums)
    assert all(len(sums[k]) <= 2 for k in order)
    rows = []
    for k in order:
        (e0, c0), (e1, c1) = (*sums[k], (0, 0.0))[:2]
        rows.append(f"{{{_lit(c0)}, {_lit(c1)}, {k << 16 | e1 << 8 | e0}, 0}}")
    out += [f"__device__ const CoupleTerm kCouple{lin}[{len(order)}] = {{" + ", ".join(rows) + "};",
            f"template <> struct TpCoupled<{lin}> {{",
            f"    static constexpr int kFloats = {stride}, kEntries = {len(order)};",
            f"    static __device__ __forceinline__ const CoupleTerm* terms() {{ return kCouple{lin}; }}",
            "};", ""]

    def t_loads(p):
        # the groups of four that start with path p (paths are not padded: a group may have begun with the path before)
        ks = [k for (pp, _, _), k in offset.items() if pp == p]
        first, last = -(-min(ks) // 4), max(ks) // 4
        lines = [f"const float4 t{k} = T[{k}];" for k in range(first, last + 1)]
        return lines, lambda mo, mi: f"t{offset[p, mo, mi] // 4}.{'xyzw'[offset[p, mo, mi] % 4]}"

    for ld in (64, 32) if lin == 1 else (64,):          # all channels, or half of them (tp_onchip.cu)
        fwd = [f"template <> __device__ __forceinline__ void tp_forward_coupled<{lin}, {ld}>(const float2* x, const float4* T, "
               f"const float2* w, float2 (&acc)[{mid}]) {{"]
        fwd += [f"    const float2 x{k} = x[{k * ld}];" for k in range(in_dim)]
        for p, path in enumerate(paths):
            l_in, l_out, off = path["l_in"], path["l_out"], path["in_off"]
            n_in, n_out = 2 * l_in + 1, 2 * l_out + 1
            loads, t = t_loads(p)
            fwd.append(f"    {' '.join(loads)}\n    {{  // path {p}: {l_in} x {path['l_edge']} -> {l_out}")
            fwd.append(f"        const float2 wp = w[{p * ld}];")
            if n_in <= n_out:
                fwd.append("        " + " ".join(f"const float2 a{mi} = __fmul2_rn(wp, x{off + mi});" for mi in range(n_in)))
            for mo in range(n_out):
                ins = [mi for mi in range(n_in) if (p, mo, mi) in offset]
                slot = slots[p, mo]
                if n_in <= n_out:
                    fwd += [f"        acc[{slot}] = __ffma2_rn(a{mi}, pair_of({t(mo, mi)}), acc[{slot}]);" for mi in ins]
                else:
                    lines = [f"float2 s = __fmul2_rn(x{off + ins[0]}, pair_of({t(mo, ins[0])}));"]
                    lines += [f"s = __ffma2_rn(x{off + mi}, pair_of({t(mo, mi)}), s);" for mi in ins[1:]]
                    fwd.append(f"        {{ {' '.join(lines)} acc[{slot}] = __ffma2_rn(wp, s, acc[{slot}]); }}")
            fwd.append("    }")
        fwd += ["}", ""]

        bwd = [f"template <> __device__ __forceinline__ void tp_backward_coupled<{lin}, {ld}>(const float2* xp, const float4* T, "
               f"const float2* w, const float2* wd, const float2 (&g)[{mid}], float2 (&dY)[16], float2& dr, float2 (&dx)[{in_dim}]) {{"]
        bwd += [f"    const float2 x{k} = xp[{k * ld}];" for k in range(in_dim)]
        for p, path in enumerate(paths):
            l_in, l_out, off = path["l_in"], path["l_out"], path["in_off"]
            n_in, n_out = 2 * l_in + 1, 2 * l_out + 1
            loads, t = t_loads(p)
            bwd.append(f"    {' '.join(loads)}\n    {{  // path {p}: {l_in} x {path['l_edge']} -> {l_out}")
            bwd.append(f"        const float2 wp = w[{p * ld}];")
            # gradient of the weighted sender features, shared by dx and by the derivative of the weight
            for mi in range(n_in):
                outs = [mo for mo in range(n_out) if (p, mo, mi) in offset]
                lines = [f"float2 u{mi} = __fmul2_rn(g[{slots[p, outs[0]]}], pair_of({t(outs[0], mi)}));"]
                lines += [f"u{mi} = __ffma2_rn(g[{slots[p, mo]}], pair_of({t(mo, mi)}), u{mi});" for mo in outs[1:]]
                bwd.append("        " + " ".join(lines))
            bwd.append("        float2 dw = __fmul2_rn(" + f"x{off}, u0); "
                       + " ".join(f"dw = __ffma2_rn(x{off + mi}, u{mi}, dw);" for mi in range(1, n_in))
                       + f" dr = __ffma2_rn(wd[{p * ld}], dw, dr);")
            bwd.append("        " + " ".join(f"dx[{off + mi}] = __ffma2_rn(wp, u{mi}, dx[{off + mi}]);" for mi in range(n_in)))
            # products of weighted features and message gradient, coupled into the harmonics' gradient
            by_pair: dict[tuple, list] = {}
            for mi, me, mo, c in path["terms"]:
                by_pair.setdefault((mi, mo), []).append((path["edge_off"] + me, c))
            weigh_in = n_in <= n_out
            if weigh_in:
                bwd.append("        " + " ".join(f"const float2 a{mi} = __fmul2_rn(wp, x{off + mi});" for mi in range(n_in)))
            else:
                bwd.append("        " + " ".join(f"const float2 a{mo} = __fmul2_rn(wp, g[{slots[p, mo]}]);" for mo in range(n_out)))
            for (mi, mo), terms in sorted(by_pair.items()):
                prod = (f"a{mi}, g[{slots[p, mo]}]" if weigh_in else f"x{off + mi}, a{mo}")
                if len(terms) == 1 and abs(terms[0][1] - 1.0) < 1e-12:
                    e = terms[0][0]
                    bwd.append(f"        dY[{e}] = __ffma2_rn({prod}, dY[{e}]);")
                else:
                    bwd.append(f"        {{ const float2 s = __fmul2_rn({prod}); "
                               + " ".join(f"dY[{e}] = __ffma2_rn(s, pair_of({_lit(c)}), dY[{e}]);" for e, c in terms) + " }")
            bwd.append("    }")
        bwd += ["}", ""]
        out += fwd + bwd
    return "\n".join(out)


def render_coupled() -> str:
    head = ["// GENERATED by fastmace_b200/codegen.py from fastmace_b200/so3.py -- do not edit.",
            "// The channelwise tensor product for two channels per thread on harmonics coupled once per edge (same",
            "// coefficients and message layout as tp_generated.cuh). x, w, wd: this thread's channel pair of the rows in",
            "// shared memory, LD pairs from one component or path to the next; T: the edge's couplings, 16-byte aligned.",
            "#pragma once",
            "",
            "namespace fmb {",
            "",
            "__device__ __forceinline__ float2 pair_of(float v) { return make_float2(v, v); }",
            "template <int LIN> struct TpCoupled;",
            "struct alignas(16) CoupleTerm { float c0, c1; int at, unused; };",
            "// LD: channel pairs from one row to the next",
            "template <int LIN, int LD> __device__ __forceinline__ void tp_forward_coupled(const float2* x, const float4* T, const float2* w, "
            "float2 (&acc)[LIN == 0 ? 16 : LIN == 1 ? 40 : 71]);",
            "template <int LIN, int LD> __device__ __forceinline__ void tp_backward_coupled(const float2* xp, const float4* T, "
            "const float2* w, const float2* wd, const float2 (&g)[LIN == 0 ? 16 : LIN == 1 ? 40 : 71], float2 (&dY)[16], "
            "float2& dr, float2 (&dx)[(LIN + 1) * (LIN + 1)]);",
            ""]
    return "\n".join(head + [_emit_coupled(lin) for lin in (0, 1, 2)] + ["}  // namespace fmb", ""])


_tp_main = main


def main() -> str:  # noqa: F811  (both generated headers)
    out = _tp_main()
    _write(SYMCON_OUT, render_symcon())
    _write(COUPLED_OUT, render_coupled())
    return out


if __name__ == "__main__":
    print(main())
