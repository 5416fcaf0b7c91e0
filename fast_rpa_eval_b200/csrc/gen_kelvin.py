"""Generates kelvin_horner.cuh: straight-line Horner evaluation of the far-field
polynomial  P(u) = sum_{a+b+c <= lam} coef(a,b,c) ux^a uy^b uz^c  for
lam = 0..8, for 1, 2 and 4 points at a time (sharing every coefficient load).

Coefficients are packed by degree first, so a coefficient's slot does not
depend on the largest degree in use and one body per lam serves every
l_pot_max: all monomials of total degree < d, then degree d by a, then b, each
(degree, a) run starting at an even slot.  Rows b and b + 1 (b even) of one a
are evaluated in lockstep by degree, so that the two coefficients of a step
are one aligned 16-byte load and the rows' chains overlap.  Within a step the
points that take the same coefficient follow one another, and the multiply-adds
are volatile so that this order reaches the hardware: three distinct 64-bit
register operands take longer to read than the FP64 pipe needs for the
operation, a repeated one does not.  Measured (20 warps per SM, coefficients in
shared memory, TFLOP/s of a peak of 37): 2 points 24.7 in the compiler's order
and 28.3 in this one; 4 points 28.3 and 30.9; 1 point 18 (two shared-memory
coefficients per multiply-add cycle).
The code is emitted rather than left to template unrolling because nvcc's
optimiser takes tens of minutes on the equivalent nested unrolled loops.

The build (fast_rpa_eval_b200/build.py) writes it into its build directory
before compiling; by hand:

    python gen_kelvin.py <output path>
"""
import os

LMAX = 8


def gidx(a, b, c):
    d = a + b + c
    off = d * (d + 1) * (d + 2) // 6
    pos = 0
    for aa in range(a):
        pos += d - aa + 1
    return off + pos + b


def slot(a, b, c):
    """Position of coef(a, b, c) in a record."""
    d = a + b + c
    off = sum((dd - aa + 2) // 2 * 2 for dd in range(d) for aa in range(dd + 1))
    return off + sum((d - aa + 2) // 2 * 2 for aa in range(a)) + b


def slots(lam):
    return slot(0, 0, lam + 1)


def horner_body(lam, npts, masked=False):
    """P[j] for npts points.  masked (one point): the degrees above the lane's
    own l_atom_max are dropped: a partial sum is multiplied on by zero instead
    of by the coordinate where all of its terms lie above it."""
    out = []
    emit = out.append
    pts = range(npts)

    def coord(v, j, deg):
        return f"(own >= {deg} ? {v}[{j}] : 0.0)" if masked else f"{v}[{j}]"

    def fma(r, u, k):
        return f"{r} = fma({r}, {u}, {k});" if masked else f"fma_ordered({r}, {u}, {k});"

    first_a = True
    for a in range(lam, -1, -1):
        rows = lam - a  # b = 0..rows
        first_b = True
        for b in range(rows // 2 * 2, -1, -2):  # rows b and b + 1
            pair = b + 1 <= rows
            emit("    {")
            for d in range(lam, a + b - 1, -1):  # degree step: c = d - a - b for row b, one less for row b + 1
                both = pair and d >= a + b + 1
                s0 = slot(a, b, d - a - b)
                if both:
                    emit(f"      {'{'} const double2 k = *reinterpret_cast<const double2 *>(c + {s0});")
                else:
                    emit(f"      {'{'} const double kx = c[{s0}];")
                kx = "k.x" if both else "kx"
                for j in pts:
                    if d == lam:
                        emit(f"        R{j} = {kx};")
                    else:
                        emit(f"        {fma(f'R{j}', coord('uz', j, d + 1), kx)}")
                for j in reversed(pts) if both else ():
                    if d == lam:
                        emit(f"        S{j} = k.y;")
                    else:
                        emit(f"        {fma(f'S{j}', coord('uz', j, d + 1), 'k.y')}")
                emit("      }")
            for j in pts:
                if pair:
                    if first_b:
                        emit(f"      Q{j} = S{j};")
                    else:
                        emit(f"      Q{j} = fma(Q{j}, {coord('uy', j, a + b + 2)}, S{j});")
                    emit(f"      Q{j} = fma(Q{j}, {coord('uy', j, a + b + 1)}, R{j});")
                elif first_b:
                    emit(f"      Q{j} = R{j};")
                else:
                    emit(f"      Q{j} = fma(Q{j}, {coord('uy', j, a + b + 1)}, R{j});")
            emit("    }")
            first_b = False
        for j in pts:
            if first_a:
                emit(f"    P[{j}] = Q{j};")
            else:
                emit(f"    P[{j}] = fma(P[{j}], {coord('ux', j, a + 1)}, Q{j});")
        first_a = False
    return "\n".join(out)


def render() -> str:
    lines = [
        "// Generated by gen_kelvin.py: straight-line Horner evaluation of the",
        "// Kelvin-inverted far-field polynomial, degree-graded coefficient packing.",
        "// Do not edit by hand.",
        "#pragma once",
        "",
        "namespace frpa {",
        "",
        f"constexpr int KELVIN_LMAX = {LMAX};",
        "// number of coefficients of degree <= L",
        "__host__ __device__ constexpr int kelvin_count(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }",
        "// doubles that the coefficients of degree <= L take in a record",
        "__host__ __device__ constexpr int kelvin_slots(int L) {",
        "  int n = 0;",
        "  for (int d = 0; d <= L; ++d)",
        "    for (int a = 0; a <= d; ++a) n += (d - a + 2) / 2 * 2;",
        "  return n;",
        "}",
        "// position of ux^a uy^b uz^c in a record",
        "__host__ __device__ constexpr int kelvin_slot(int a, int b, int c) {",
        "  int n = kelvin_slots(a + b + c - 1) + b;",
        "  for (int aa = 0; aa < a; ++aa) n += (a + b + c - aa + 2) / 2 * 2;",
        "  return n;",
        "}",
        "// r = r u + k, in program order with its neighbours",
        "__device__ __forceinline__ void fma_ordered(double &r, double u, double k) {",
        '  asm volatile("fma.rn.f64 %0, %0, %1, %2;" : "+d"(r) : "d"(u), "d"(k));',
        "}",
        "// index of ux^a uy^b uz^c among the coefficients (by degree, a, b; no padding)",
        "__host__ __device__ constexpr int kelvin_index(int a, int b, int c) {",
        "  return (a + b + c) * (a + b + c + 1) * (a + b + c + 2) / 6 + a * (a + b + c + 1) - a * (a - 1) / 2 + b;",
        "}",
        "",
    ]
    # check the closed form used above against gidx
    for d in range(LMAX + 1):
        for a in range(d + 1):
            for b in range(d - a + 1):
                c = d - a - b
                assert slot(a, b, c) % 2 == b % 2 and slot(a, b, c) < slots(d)
                closed = d * (d + 1) * (d + 2) // 6 + a * (d + 1) - a * (a - 1) // 2 + b
                assert closed == gidx(a, b, c), (a, b, c)
    for npts in (1, 2, 4):
        for lam in range(LMAX + 1):
            lines.append(f"__device__ __forceinline__ void kelvin_horner_{lam}_{npts}(const double *__restrict__ c, "
                         f"const double *ux, const double *uy, const double *uz, double *P) {{")
            lines.append("  " + " ".join(f"double Q{j}, R{j}, S{j};" for j in range(npts)))
            lines.append(horner_body(lam, npts))
            lines.append("}")
            lines.append("")
        lines.append(f"__device__ __forceinline__ void kelvin_eval_{npts}(int lam, const double *__restrict__ c, "
                     "const double *ux, const double *uy, const double *uz, double *P) {")
        lines.append("  switch (lam) {")
        for lam in range(LMAX + 1):
            lines.append(f"    case {lam}: kelvin_horner_{lam}_{npts}(c, ux, uy, uz, P); break;")
        lines.append("    default: break;")
        lines.append("  }")
        lines.append("}")
        lines.append("")
    for lam in range(LMAX + 1):
        lines.append(f"__device__ __forceinline__ void kelvin_masked_{lam}(const double *__restrict__ c, "
                     "const double *ux, const double *uy, const double *uz, int own, double *P) {")
        lines.append("  double Q0, R0, S0;")
        lines.append(horner_body(lam, 1, masked=True))
        lines.append("}")
        lines.append("")
    lines.append("// degree `lam` (uniform over the warp), of which this lane keeps the degrees up to `own` <= lam; the")
    lines.append("// dropped partial sums must be finite")
    lines.append("__device__ __forceinline__ void kelvin_masked_eval(int lam, const double *__restrict__ c, "
                 "const double *ux, const double *uy, const double *uz, int own, double *P) {")
    lines.append("  switch (lam) {")
    for lam in range(LMAX + 1):
        lines.append(f"    case {lam}: kelvin_masked_{lam}(c, ux, uy, uz, own, P); break;")
    lines.append("    default: break;")
    lines.append("  }")
    lines.append("}")
    lines.append("")
    lines.append("// kelvin_eval<N>: N points at a time")
    lines.append("template <int N>")
    lines.append("__device__ __forceinline__ void kelvin_eval(int lam, const double *__restrict__ c, const double *ux, "
                 "const double *uy, const double *uz, double *P);")
    for npts in (1, 2, 4):
        lines.append("template <>")
        lines.append(f"__device__ __forceinline__ void kelvin_eval<{npts}>(int lam, const double *__restrict__ c, "
                     "const double *ux, const double *uy, const double *uz, double *P) {")
        lines.append(f"  kelvin_eval_{npts}(lam, c, ux, uy, uz, P);")
        lines.append("}")
    lines.append("")
    lines.append("}  // namespace frpa")
    lines.append("")
    return "\n".join(lines)


def write(dst: str) -> None:
    text = render()
    if os.path.exists(dst) and open(dst).read() == text:
        return
    with open(dst, "w") as f:
        f.write(text)


if __name__ == "__main__":
    import sys

    write(sys.argv[1])
