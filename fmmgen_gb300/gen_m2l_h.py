"""Generate fmmgen_gb300/csrc/m2l_h_{f32,f64}_p{P}.cu: M2L kernels over harmonic coefficients, FP32 and FP64.

The derivatives D_k of 1/R are harmonic: D_{k+2ez} = -D_{k+2ex} - D_{k+2ey}.  In
    L^_n = sum_m D_{n+m} rho^|m| M~_m,     |n| + |m| <= q
(the contraction of fmmgen/expansions.py:144-172; see csrc/eval.cu for the scaling) the multipole terms with m_z >= 2 can
therefore be added into those with m_z in {0, 1} of the same degree beforehand,
    M'_(a,b,e) = sum_j (-1)^j sum_i C(j,i) M~_(a-2i, b-2(j-i), e+2j),
and the outputs with n_z >= 2 follow from those with n_z in {0, 1} afterwards,
    L_(a,b,e+2j) = (-1)^j sum_i C(j,i) L_(a+2i, b+2(j-i), e).
(p+1)^2 instead of (p+1)(p+2)(p+3)/6 coefficients on each side: at p = 8 1,365 multiply-adds per pair instead of 3,003,
at p = 12 5,551 instead of 18,564, and about half the bytes per source row.  Both foldings keep the degree, so truncating
a pair at its own order q keeps the terms |n| + |m| <= q as before.  The operator vectors hold the D_k with k_z <= 2.

Layouts, degree by degree: coefficients (h_index) k_z = 0 then 1, x descending; operators (d_index) k_z = 0, 1, 2.

A thread takes one target cell and a slice of its list (csrc/m2l_h.cuh has the pair loop's pieces); its outputs stay in
registers.  Per pair the warp copies the 32 lanes' source and operator rows into shared memory with asynchronous copies,
eight lanes per row so that each copy instruction covers whole 128-byte lines, a pair ahead of the multiply-adds.  FP32:
the source row moves into registers and its buffer is refilled at once; the operator is read as 16-byte words.  FP64: the
FP64 pipe issues one warp instruction per 16 clocks of an SM, so the source row stays in shared memory and each
multiply-add loads its own operand.  Every index is resolved here; the terms are nested by the degree of k so that a lane
stops at its pair's order.  Outputs with many terms per pair sum a pair's terms first (rounding grows with the pairs).

A family covers every order up to its largest.  Orders above 8 split the (output degrees) x (multipole degrees) square
into parts whose registers and staged rows leave eight warps per SM; the first part of a group of outputs stores, the
others add.
"""
import os

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
FAMILIES = [4, 6, 8, 12]
TYPES = [("f32", "float", 4), ("f64", "double", 8)]
PARTIAL_MIN_TERMS = 21  # outputs with at least this many terms per pair sum per pair first
SMEM = 227 * 1024       # shared memory of a block


def h_terms(d):
    """Coefficients up to degree d."""
    return (d + 1) * (d + 1) if d >= 0 else 0


def d_terms(d):
    """Operator entries up to degree d."""
    return 0 if d < 0 else 1 + 3 * d * (d + 1) // 2


def multiply_adds(q):
    """Multiply-adds of a pair at order q, whatever the family and the source order."""
    return sum((2 * n + 1) * (2 * m + 1) for n in range(q + 1) for m in range(q + 1 - n))


def coeffs(p):
    """The coefficient indices (x, y, z), z <= 1, in layout order."""
    return [(x, d - z - x, z) for d in range(p + 1) for z in range(min(d, 1) + 1) for x in range(d - z, -1, -1)]


def operators(p):
    return [(x, d - z - x, z) for d in range(p + 1) for z in range(min(d, 2) + 1) for x in range(d - z, -1, -1)]


def parts(pmax):
    """(first and last output degree, first and last multipole degree, stores) of each kernel of a family."""
    if pmax <= 8:
        return [(0, pmax, 0, pmax, True)]
    return [(0, 4, 0, 6, True), (0, 4, 7, 8, False), (0, 4, 9, 12, False), (5, 7, 0, 4, True), (5, 7, 5, 7, False),
            (8, 12, 0, 4, True)]


def plan(pmax):
    """The kernels of a family: outs, temps and terms [(degree, k, n, m)] sorted, as layout indices."""
    co, op = coeffs(pmax), {k: i for i, k in enumerate(operators(pmax))}
    out = []
    for n0, n1, m0, m1, first in parts(pmax):
        terms = []
        for i in range(h_terms(n0 - 1), h_terms(n1)):
            for j in range(h_terms(m0 - 1), h_terms(m1)):
                n, m = co[i], co[j]
                d = sum(n) + sum(m)
                if d <= pmax:
                    terms.append((d, op[(n[0] + m[0], n[1] + m[1], n[2] + m[2])], i, j))
        terms.sort()
        cnt = {}
        for _, _, i, _ in terms:
            cnt[i] = cnt.get(i, 0) + 1
        out.append(dict(n=(n0, n1), m=(m0, m1), first=first, dmin=n0 + m0, dmax=max(t[0] for t in terms),
                        outs=list(range(h_terms(n0 - 1), h_terms(n1))), terms=terms,
                        temps=sorted(i for i, v in cnt.items() if v >= PARTIAL_MIN_TERMS)))
    return out


def geometry(kern, size):
    """16-byte words of the staged rows: (first, end, row stride) of the source and of the operator, and the
    operator word at which the second stage begins (about half of the multiply-adds on each side)."""
    per = 16 // size

    def rng(lo, hi):
        q0 = lo // per & ~1  # rows start on a 32-byte sector
        q1 = -(-hi // per)
        return q0, q1, (q1 - q0) | 1  # an odd stride: the lanes' 16-byte reads fall in distinct banks

    mq = rng(h_terms(kern["m"][0] - 1), h_terms(kern["m"][1]))
    dq = rng(d_terms(kern["dmin"] - 1), d_terms(kern["dmax"]))
    half, seen, split = len(kern["terms"]) / 2, 0, dq[0] + 8
    for q in range(dq[0] + 8, dq[1], 8):
        seen = sum(1 for t in kern["terms"] if t[1] // per < q)
        split = q
        if seen >= half:
            break
    return mq, dq, min(split, dq[1])


def operator_pieces(mq, dq, nout):
    """FP64: one warp a scheduler cannot keep the pipe busy, and a whole operator beside the source row often leaves no
    room for more (p = 8: 49 KB a warp, four warps an SM, the pipe 74 % busy).  The pieces in which the operator
    is brought in instead, one after the other through one buffer, and the buffer's row stride: the fewest that fit
    eight warps; None where the whole fits them, or no pieces do.  10^6 charges, p = 8: 48.9 -> 37.1 ms; 1.1 M pairs of
    dipoles, p = 6: 1.38 -> 1.33 ms."""
    room = 56  # 16-byte words of a lane's row: 8 x 32 x 16 x 56 = 224 KB
    if mq[2] + dq[2] <= room or -(-nout * 8 // 16) > room:
        return None
    for n in range(2, 7):
        size = -(-(dq[1] - dq[0]) // n) + 1 & ~1  # pieces start on a 32-byte sector
        if mq[2] + (size | 1) <= room:
            return [(q, min(q + size, dq[1])) for q in range(dq[0], dq[1], size)], size | 1
    return None


def emit(pmax, ki, kern, tag, typ, size):
    per = 16 // size
    mq, dq, split = geometry(kern, size)
    f32 = typ == "float"
    name = f"k_m2lh_{tag}_p{pmax}_{ki}"
    i0, temps, dmin = kern["outs"][0], set(kern["temps"]), kern["dmin"]
    degs = [sum(c) for c in coeffs(pmax)]
    n0, m0, m1 = kern["n"][0], kern["m"][0], kern["m"][1]
    cut = None if f32 else operator_pieces(mq, dq, len(kern["outs"]))
    pieces, dstride = cut or ([(dq[0], split), (split, dq[1])], dq[2])
    words = max(mq[2] + dstride, -(-len(kern["outs"]) * size // 16) if cut else 0)  # the sums go there in the end
    used = sorted({j for _, _, _, j in kern["terms"]})
    L = [f"// outputs of degree {kern['n'][0]}..{kern['n'][1]}, multipole degrees {m0}..{m1}: {len(kern['outs'])} "
         f"accumulators, {len(temps)} per-pair sums, {len(kern['terms'])} multiply-adds at order {pmax}",
         f"__global__ void __launch_bounds__(256, 1) {name}(const HParams<{typ}> P) {{",
         "  extern __shared__ float4 h_smem[];",
         "  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;",
         f"  float4 *const mb = h_smem + w * {32 * words}, *const db = mb + {32 * mq[2]};",
         f"  const H{'F32' if f32 else 'F64'}Row<{mq[2]}, {dstride}> row(mb, db, lane);",
         "  HList it(P, lane, w, W);"]
    L.append("  " + typ + " " + ", ".join(f"a{i - i0} = 0" for i in kern["outs"]) + ";")

    def stage(what, lo, hi, base, stride, deg, terms, qvar, rowvar, src, rowlen, ind):
        # the words [lo, hi) of the lanes' rows, as far as order qvar needs them
        return (f"{ind}h_stage<{lo}, {hi}, {base}, {stride}>({what}, {src}, {rowlen}, {rowvar}, lane, "
                f"h_words<{size}>({terms}({deg})));")

    def stage_m(qvar, rowvar, ind):
        return stage("mb", mq[0], mq[1], mq[0], mq[2], f"min({m1}, {qvar} - {n0})", "h_terms", qvar, rowvar, "P.M",
                     "P.mstr", ind)

    def stage_d(half, qvar, rowvar, ind):
        lo, hi = pieces[half]
        if lo >= hi:
            return ""
        return stage("db", lo, hi, lo if cut else dq[0], dstride, f"min({kern['dmax']}, {qvar})", "h_dterms", qvar, rowvar, "P.D",
                     "P.dstr", ind)

    L.append(f"  if (it.begin({dmin})) {{")
    for s in (stage_m("it.qmax", "it.B", "    "), stage_d(0, "it.qmax", "it.c", "    "), None,
              "" if cut else stage_d(1, "it.qmax", "it.c", "    ")):
        L.append("    h_commit();" if s is None else s)
    L += ["    h_commit();", "  }"]
    L.append("  while (it.on_any) {")
    L.append(f"    it.look_ahead({dmin}{f', fmm_wide_levels({pmax})' if f32 else ''});")
    L.append("    const int ql = it.ql;")
    if f32:
        L.append("    h_wait<1>();  // the source row and the operator's first half")
        L.append("    __syncwarp();")
        for q in range(mq[0], mq[1]):
            if any(j // per == q for j in used):
                L.append(f"    const float4 mq{q} = row.m({q - mq[0]});")
        L.append("    float " + ", ".join(f"m{j} = mq{j // per}.{'xyzw'[j % per]}" for j in used) + ";")
        sc = sorted({degs[j] for j in used if degs[j] > 0})
        L.append("    if (it.rescale) {")
        for d in sc:
            L.append(f"      const float s{d} = h_exp2<float>({d} * it.dl);")
            L.append("      " + " ".join(f"m{j} *= s{d};" for j in used if degs[j] == d))
        L.append("    }")
        L.append("    __syncwarp();")
        L.append("    if (it.on_next)")
        L.append(stage_m("it.qmaxn", "it.Bs", "      "))
        L.append("    h_commit();")
    else:
        L.append("    h_wait<0>();")
        L.append("    __syncwarp();")
        sc = sorted({degs[j] for j in used if degs[j] > 0})
        L.append("    if (it.rescale) {  // the lane's own row")
        for d in sc:
            js = [j for j in used if degs[j] == d]
            L.append(f"      row.scale({js[0] - mq[0] * per}, {js[-1] + 1 - mq[0] * per}, h_exp2<double>({d} * it.dl));")
        L.append("    }")
        L.append("    __syncwarp();")
    if temps:
        L.append("    " + typ + " " + ", ".join(f"t{i - i0} = 0" for i in sorted(temps)) + ";")

    def block(lo, hi):
        by = {}
        for t in kern["terms"]:
            if lo <= t[1] // per < hi:
                by.setdefault(t[0], []).append(t)
        depth, loaded = 0, set()
        for d in sorted(by):
            L.append("    " + "  " * depth + f"if (ql >= {d}) {{")
            depth += 1
            ind = "    " + "  " * depth
            line = []
            for _, k, i, j in by[d]:
                acc = f"t{i - i0}" if i in temps else f"a{i - i0}"
                if f32:
                    if k // per not in loaded:
                        loaded.add(k // per)
                        line.append(f"const float4 d{k // per} = row.d({k // per - dq[0]});")
                    line.append(f"{acc} = fmaf(d{k // per}.{'xyzw'[k % per]}, m{j}, {acc});")
                else:
                    if k not in loaded:
                        loaded.add(k)
                        line.append(f"const double d{k} = row.d({k - (lo if cut else dq[0]) * per});")
                    line.append(f"row.fma<{j - mq[0] * per}>({acc}, d{k});")
                if len(line) >= 4:
                    L.append(ind + " ".join(line))
                    line = []
            if line:
                L.append(ind + " ".join(line))
        for k in range(depth, 0, -1):
            L.append("    " + "  " * (k - 1) + "}")

    if cut:
        for n, (lo, hi) in enumerate(pieces):
            if n:  # the other warps multiply meanwhile
                L.append("    __syncwarp();")
                L.append(stage_d(n, "it.qmax", "it.c", "    "))
                L += ["    h_commit();", "    h_wait<0>();", "    __syncwarp();"]
            block(lo, hi)
    else:
        block(dq[0], split)
        L.append("    __syncwarp();")
        L.append("    if (it.on_next)")
        L.append(stage_d(0, "it.qmaxn", "it.cs", "      "))
        L.append("    h_commit();")
        if f32:
            L.append("    h_wait<2>();  // the operator's second half")
            L.append("    __syncwarp();")
        block(split, dq[1])
    if temps:
        L.append("    " + " ".join(f"a{i - i0} += t{i - i0};" for i in sorted(temps)))
    L.append("    __syncwarp();")
    L.append("    if (it.on_next) {")
    if not f32:
        L.append(stage_m("it.qmaxn", "it.Bs", "      "))
    s = stage_d(0 if cut else 1, "it.qmaxn", "it.cs", "      ")
    if s:
        L.append(s)
    L.append("    }")
    L.append("    h_commit();")
    L.append("    it.advance();")
    L.append("  }")
    L.append("  h_wait<0>();")
    L.append("  // the warps' sums, in shared memory")
    L.append(f"  {typ} *const sum = ({typ} *)(h_smem + w * {32 * words}) + lane;")
    L.append("  __syncwarp();")
    for k in range(0, len(kern["outs"]), 4):
        L.append("  " + " ".join(f"sum[{32 * (i - i0)}] = a{i - i0};" for i in kern["outs"][k:k + 4]))
    assert len(kern["outs"]) * size <= 16 * words
    L.append(f"  h_store<{typ}, {len(kern['outs'])}, {16 * 32 * words // size}, {'false' if kern['first'] else 'true'}>"
             f"(P, ({typ} *)h_smem, {i0}, W);")
    L.append("}")
    return name, dmin, 16 * 32 * words, "\n".join(L)


def family_file(tag, pmax):
    return f"m2l_h_{tag}_p{pmax}.cu"


def generate_family(tag, typ, size, pmax):
    P = [f"// {family_file(tag, pmax)} -- generated by fmmgen_gb300/gen_m2l_h.py; do not edit.",
         f"// M2L over harmonic coefficients in {typ}, orders up to {pmax} (see m2l_h.cuh).", '#include "m2l_h.cuh"', ""]
    table = []
    for ki, kern in enumerate(plan(pmax)):
        name, dmin, smem, code = emit(pmax, ki, kern, tag, typ, size)
        P += [code, ""]
        table.append((name, dmin, smem))
    P.append(f"int fmm_m2lh_{tag}_p{pmax}(const HParams<{typ}> &P, cudaStream_t st) {{")
    for name, dmin, smem in table:
        P.append(f"  if (P.p >= {dmin})")
        P.append(f"    if (int rc = h_launch({name}, P, {smem}, {min(8, SMEM // smem)}, st)) return rc;")
    P += ["  return FMM_OK;", "}"]
    with open(os.path.join(CSRC, family_file(tag, pmax)), "w") as f:
        f.write("\n".join(P) + "\n")


def generate():
    for tag, typ, size in TYPES:
        for pmax in FAMILIES:
            generate_family(tag, typ, size, pmax)


def outputs():
    return [os.path.join(CSRC, family_file(tag, pmax)) for tag, _, _ in TYPES for pmax in FAMILIES]


if __name__ == "__main__":
    generate()
    for o in outputs():
        print(o)
