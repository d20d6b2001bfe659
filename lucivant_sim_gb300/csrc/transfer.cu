// Lowering of real64 (Pauli-transfer) register blocks.
//
// A noisy one-qubit gate is a real 4x4 operator with first row (1, 0, 0, 0): nine products and, for
// amplitude damping, a shift of Z, 10 multiply-adds per four coefficients, on a GPU whose FP64 units
// run 2 a clock and SM. Its 3x3 part is written as
//   M = S * W * V,   V and S on the pair (X, Y), W on the pair (X, Z),
// each pair map as two shears with unit diagonal, [[1, p], [q, 1]], after an exchange of the pair
// where that keeps the pivot the larger product. The scales left over move to one side and merge
// into a diagonal of the block, there already for the two-qubit gate's noise. That is 6
// multiply-adds and the shift. A gate and phase-covariant noise on a qubit that controls the next cx
// needs no S: its rotation about Z commutes with all that and is multiplied into the qubit's next
// operator, on the host: 4 and the shift. Measured (12 qubits, 12 layers of noisy u3 and cx, 64
// noise models): 426 -> 286 multiply-adds a coefficient, 610 -> 416 ms, FP64 units 90% busy before
// and after; 9 qubits, 20 layers, 8 models, interpreted passes: 3.25 -> 2.28 ms.
//
// A coefficient's error is common to all it multiplies, so each is formed as a pair of doubles and
// rounded once. Measured, 6 qubits x 20 layers, 12 models, against the operators as given in 80 bits:
// 6.0e-16 for the dense products, 1.14e-15 with coefficients formed in double precision, 6.9e-16 now.
//
// Decided per member from its own data or from the operators' structure, so a member of a batch gets
// the arithmetic it would get by itself. A member whose operator does not factor well (a reset, full
// dephasing) keeps the dense rows.
#include <algorithm>
#include <cmath>

#include "../../include/lsg.h"
#include "transfer.cuh"
#include "two.cuh"

namespace lsg {

namespace {

// Entries this small beside an operator's largest are the rounding of zero (products of gate matrices).
constexpr double kZero = 1e-15;
// Pivot ratios beyond this keep the dense form.
constexpr double kSteep = 64.0;

enum { Z = 1, X = 2, Y = 3 };

struct Mat4 {
    Two a[4][4];
};
struct Pair {  // rows (a, b), (c, d)
    Two a, b, c, d;
};

bool is_transfer(const TileOp& t) { return t.tmpl >= kT_TPD2 && t.tmpl < kT_TPD2 + 16; }
bool is_rename(int code) { return code >= kT_X1 && code < kT_SWAP + 16; }
bool is_diagonal(const TileOp& t) { return t.tmpl == kT_DIAG || t.tmpl == kT_SCALE; }

// (entries that move_outer_rotations appended have their rounding errors in `low`)
Mat4 matrix_of(const TileOp& t, const Pool& pool, int64_t b) {
    const int64_t at = 2 * (t.data + (t.stride ? b * t.stride : 0));
    Mat4 m;
    for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c) {
            const int64_t i = at + 2 * (4 * r + c);
            m.a[r][c] = Two(pool.data[i], i < pool.own ? 0.0 : pool.low[i - pool.own]);
        }
    return m;
}

Mat4 mul(const Mat4& x, const Mat4& y) {
    Mat4 m;
    for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c) {
            Two s = x.a[r][0] * y.a[0][c];
            for (int k = 1; k < 4; ++k) s = s + x.a[r][k] * y.a[k][c];
            m.a[r][c] = s;
        }
    return m;
}

double largest(const Mat4& m) {
    double big = 0.0;
    for (int r = 1; r < 4; ++r)
        for (int c = 1; c < 4; ++c) big = std::max(big, std::fabs(m.a[r][c].v));
    return big;
}

// The inverse of S on rows (X, Y): its second row leaves Y without Z, its first row leaves X parallel to
// Z in the columns (X, Y). Rows of unit length. False when they are not defined well.
bool outer_inverse(const Mat4& m, double big, Pair* out) {
    const Two xz = m.a[X][Z], yz = m.a[Y][Z], h = root(xz * xz + yz * yz);
    const Two ca = m.a[X][X] * m.a[Z][Y] - m.a[X][Y] * m.a[Z][X];
    const Two cb = m.a[Y][X] * m.a[Z][Y] - m.a[Y][Y] * m.a[Z][X];
    const Two g = root(ca * ca + cb * cb);
    if (!(h.v > 1e-6 * big) || !(g.v > 1e-6 * big * big)) return false;
    Pair s{tidy(cb / g), tidy(-ca / g), tidy(-yz / h), tidy(xz / h)};
    if (s.a.v < 0.0) s.a = -s.a, s.b = -s.b;
    if (s.d.v < 0.0) s.c = -s.c, s.d = -s.d;
    // a rotation to rounding is one (with a quarter turn, either sign of its zero cosine is)
    if (std::fabs(s.b.v - s.c.v) <= kZero && std::fabs(s.a.v) <= kZero && std::fabs(s.d.v) <= kZero) s.b = -s.b;
    if (std::fabs(s.a.v - s.d.v) <= 4.0 * kZero && std::fabs(s.b.v + s.c.v) <= 4.0 * kZero) s.a = s.d, s.b = -s.c;
    if (std::fabs(s.b.v) <= kZero && std::fabs(s.c.v) <= kZero) s = Pair{1.0, 0.0, 0.0, 1.0};
    *out = s;
    return true;
}
bool is_rotation(const Pair& s) { return s.a.v == s.d.v && s.b.v == -s.c.v; }

// f = [[1, p], [q, 1]] * diag(x, y), the pair exchanged between them when `flip`; or, from the left,
// diag(x, y) * [[1, p], [q, 1]] after the exchange.
struct Shears {
    Two p, q, x = 1.0, y = 1.0;
    bool flip = false, ok = true;
};
Shears shears(Pair f, bool left) {
    Shears s;
    s.flip = std::fabs(f.a.v * f.d.v) < std::fabs(f.b.v * f.c.v);
    if (s.flip) f = Pair{f.b, f.a, f.d, f.c};
    s.p = tidy(f.b / (left ? f.a : f.d));
    s.q = tidy(f.c / (left ? f.d : f.a));
    s.x = s.flip && !left ? f.d : f.a;
    s.y = s.flip && !left ? f.a : f.d;
    s.ok = std::fabs(s.p.v) <= kSteep && std::fabs(s.q.v) <= kSteep && s.x.v != 0.0 && s.y.v != 0.0;
    return s;
}

struct Factors {
    int parts = 0;
    double v[2] = {0, 0}, w[2] = {0, 0}, s[2] = {0, 0}, shift[3] = {0, 0, 0};  // shift: Z, X, Y
    Two scale[4] = {1.0, 1.0, 1.0, 1.0};                                       // by row of the 4x4 operator
};

// m as shears with its scales before them (or, `left`, after them). Parts kTrDense when it does not
// factor to rounding.
Factors factor(const Mat4& m, bool left) {
    Factors f;
    auto dense = [&] {
        Factors d;
        d.parts = kTrDense;
        return d;
    };
    const double big = largest(m);
    if (!(big > 0.0) || !std::isfinite(big)) return dense();
    Pair si{1.0, 0.0, 0.0, 1.0}, v{m.a[X][X], m.a[X][Y], m.a[Y][X], m.a[Y][Y]}, w{1.0, 0.0, 0.0, m.a[Z][Z]};
    const double coupled = std::max({std::fabs(m.a[X][Z].v), std::fabs(m.a[Y][Z].v), std::fabs(m.a[Z][X].v), std::fabs(m.a[Z][Y].v)});
    if (coupled > kZero * big) {
        if (!outer_inverse(m, big, &si)) return dense();
        Two n[4][4];
        for (int c = Z; c <= Y; ++c) {
            n[X][c] = si.a * m.a[X][c] + si.b * m.a[Y][c];
            n[Y][c] = si.c * m.a[X][c] + si.d * m.a[Y][c];
            n[Z][c] = m.a[Z][c];
        }
        const Two nx = n[X][X] * n[X][X] + n[X][Y] * n[X][Y], nz = n[Z][X] * n[Z][X] + n[Z][Y] * n[Z][Y];
        const int from = nx.v >= nz.v ? X : Z;
        const Two h = root(from == X ? nx : nz), ux = n[from][X] / h, uy = n[from][Y] / h;
        v = Pair{ux, uy, n[Y][X], n[Y][Y]};
        w = Pair{n[X][X] * ux + n[X][Y] * uy, n[X][Z], n[Z][X] * ux + n[Z][Y] * uy, n[Z][Z]};
    }
    const Two det = si.a * si.d - si.b * si.c;
    if (!(std::fabs(det.v) > 1.0 / kSteep)) return dense();
    const Pair s{si.d / det, -si.b / det, -si.c / det, si.a / det};
    {  // the product stands for m to rounding
        const Two wv[4][4] = {{}, {Two(), w.d, w.c * v.a, w.c * v.b}, {Two(), w.b, w.a * v.a, w.a * v.b}, {Two(), Two(), v.c, v.d}};
        for (int c = Z; c <= Y; ++c) {
            const Two x = s.a * wv[X][c] + s.b * wv[Y][c], y = s.c * wv[X][c] + s.d * wv[Y][c];
            const double off = std::max({std::fabs(x.v - m.a[X][c].v), std::fabs(y.v - m.a[Y][c].v), std::fabs(wv[Z][c].v - m.a[Z][c].v)});
            if (!(off <= 4.0 * kZero * big)) return dense();
        }
    }
    Shears a, b, e;  // V, W, S
    if (!left) {
        e = shears(s, false);
        b = shears(Pair{w.a * e.x, w.b * e.x, w.c, w.d}, false);
        a = shears(Pair{v.a * b.x, v.b * b.x, v.c * e.y, v.d * e.y}, false);
        f.scale[X] = a.x, f.scale[Y] = a.y, f.scale[Z] = b.y;
    } else {
        a = shears(v, true);
        b = shears(Pair{w.a * a.x, w.b, w.c * a.x, w.d}, true);
        e = shears(Pair{s.a * b.x, s.b * a.y, s.c * b.x, s.d * a.y}, true);
        f.scale[X] = e.x, f.scale[Y] = e.y, f.scale[Z] = b.y;
    }
    if (!a.ok || !b.ok || !e.ok) return dense();
    auto part = [&](const Shears& h, int bit, int flip, double* to) {
        to[0] = h.p.value(), to[1] = h.q.value();
        if (h.flip || to[0] != 0.0 || to[1] != 0.0) f.parts |= bit | (h.flip ? flip : 0);
    };
    part(a, kTrV, kTrFlipV, f.v);
    part(b, kTrW, kTrFlipW, f.w);
    part(e, kTrS, kTrFlipS, f.s);
    for (int r = Z; r <= Y; ++r) {
        f.shift[r - 1] = (left ? m.a[r][0] / f.scale[r] : m.a[r][0]).value();
        if (m.a[r][0].value() != 0.0) f.parts |= r == Z ? kTrShiftZ : kTrShiftXY;
    }
    for (int r = Z; r <= Y; ++r)
        if (!std::isfinite(f.scale[r].v) || !std::isfinite(f.shift[r - 1])) return dense();
    return f;
}

// out[e] = f[b][e] * in[src[e]]: the renames and diagonals of a stretch of a block.
struct Composite {
    int D;
    std::vector<int> src;
    std::vector<double> f;
    Composite(int64_t members, int d) : D(d), src((size_t)d), f((size_t)(members * d), 1.0) {
        for (int e = 0; e < d; ++e) src[(size_t)e] = e;
    }
};

int rename_source(int code, int U, int e) {
    auto bit = [&](int P) { return 1 << (U - 1 - P); };
    if (code < kT_CX) return e ^ bit(code - kT_X1);
    if (code < kT_SWAP) return (e & bit((code - kT_CX) / 4)) ? e ^ bit((code - kT_CX) % 4) : e;
    const int x = bit((code - kT_SWAP) / 4), y = bit((code - kT_SWAP) % 4);
    return ((e & x) != 0) != ((e & y) != 0) ? e ^ x ^ y : e;
}

int diag_entry(const TileOp& t, int U, int e) {
    int j = 0;
    for (int i = 0; i < t.k; ++i) j = (j << 1) | ((e >> (U - 1 - t.pos[i])) & 1);
    return j;
}

unsigned positions(const TileOp& t) {
    unsigned bits = 0;
    for (int i = 0; i < t.k; ++i) bits |= 1u << t.pos[i];
    return bits;
}

template <typename T>
void permute(std::vector<T>& v, int64_t members, int U, int code) {
    const int D = 1 << U;
    std::vector<T> w(v.size());
    for (int64_t b = 0; b < members; ++b)
        for (int e = 0; e < D; ++e) w[(size_t)(b * D + e)] = v[(size_t)(b * D + rename_source(code, U, e))];
    v.swap(w);
}

template <typename T>
void times_diagonal(std::vector<T>& v, int64_t members, int U, const TileOp& t, const double* pool) {
    const int D = 1 << U;
    for (int64_t b = 0; b < members; ++b) {
        const double* p = pool + 2 * (t.data + (t.stride ? b * t.stride : 0));
        for (int e = 0; e < D; ++e) v[(size_t)(b * D + e)] = v[(size_t)(b * D + e)] * T(p[2 * diag_entry(t, U, e)]);
    }
}

// How member b's rotation of (X, Y), on positions P0, P1, passes the composite: +1 as it is, -1 the
// other way round, 0 not.
int passes(const Composite& c, int64_t b, int U, int P0, int P1) {
    const int B0 = 1 << (U - 1 - P0), B1 = 1 << (U - 1 - P1);
    int sign = 0;
    for (int e = 0; e < c.D; ++e) {
        const int s = c.src[(size_t)e];
        if (!(e & B0)) {
            if (s & B0) return 0;
            continue;
        }
        if (e & B1) continue;
        const int y = e | B1, sy = c.src[(size_t)y];
        if (!(s & B0) || (s ^ sy) != B1) return 0;
        const double fx = c.f[(size_t)(b * c.D + e)], fy = c.f[(size_t)(b * c.D + y)];
        const double near = 2.0 * kZero * std::fabs(fx);
        const int way = std::fabs(fx - fy) <= near ? 1 : std::fabs(fx + fy) <= near ? -1 : 0;
        const int turn = s & B1 ? -way : way;  // X and Y exchanged: a rotation the other way round
        if (turn == 0 || (sign && turn != sign)) return 0;
        sign = turn;
    }
    return sign;
}

}  // namespace

void move_outer_rotations(Plan& plan, int64_t batch, std::vector<double>& pool, std::vector<double>& low, Choices& form) {
    const int64_t own = (int64_t)pool.size();
    struct Touch {
        int op, pass, block;
    };
    std::vector<Touch> at[64];  // the operators on each register bit, in execution order
    auto reg = [](const PassDesc& pd, int lb) { return lb < pd.L ? lb : pd.hi[lb - pd.L]; };
    for (size_t pi = 0; pi < plan.passes.size(); ++pi) {
        const PassDesc& pd = plan.passes[pi];
        for (int bi = pd.first_block; bi < pd.first_block + pd.nblocks; ++bi) {
            const BlockDesc& blk = plan.blocks[(size_t)bi];
            for (int o = pd.first_op + blk.first; o < pd.first_op + blk.first + blk.nops; ++o)
                for (int i = 0; i < plan.ops[(size_t)o].k; ++i)
                    at[reg(pd, plan.ops[(size_t)o].lb[i])].push_back(Touch{o, (int)pi, blk.generic ? -1 : bi});
        }
    }
    for (int r0 = 0; r0 < 64; ++r0)
        for (size_t i = 0; i < at[r0].size(); ++i) {
            const Touch from = at[r0][i];
            TileOp& t = plan.ops[(size_t)from.op];
            const PassDesc& pf = plan.passes[(size_t)from.pass];
            if (from.block < 0 || !is_transfer(t) || reg(pf, t.lb[0]) != r0) continue;
            const int r1 = reg(pf, t.lb[1]);
            // the next operator on this qubit of the same kind, and the block of all between
            size_t j = i + 1;
            while (j < at[r0].size() && !is_transfer(plan.ops[(size_t)at[r0][j].op])) ++j;
            if (j == at[r0].size()) continue;
            const Touch to = at[r0][j];
            TileOp& n = plan.ops[(size_t)to.op];
            const PassDesc& pn = plan.passes[(size_t)to.pass];
            if (to.block < 0 || reg(pn, n.lb[0]) != r0 || reg(pn, n.lb[1]) != r1) continue;
            bool near = true;
            for (int r : {r0, r1})
                for (const Touch& x : at[r])
                    near = near && !(x.op > from.op && x.op < to.op && x.block != to.block);
            if (!near) continue;
            const BlockDesc& blk = plan.blocks[(size_t)to.block];
            const int U = blk.u;
            const unsigned ours = positions(n);
            Composite c(batch, 1 << U);
            unsigned shut = 0;  // positions that an operator left out has changed
            bool ok = true, each = t.stride || n.stride;
            const int begin = from.block == to.block ? from.op + 1 : pn.first_op + blk.first;
            for (int o = begin; o < to.op && ok; ++o) {
                const TileOp& x = plan.ops[(size_t)o];
                const unsigned bits = positions(x);
                if (!(is_rename(x.tmpl) || is_diagonal(x)) || (bits & shut)) {
                    ok = !(bits & ours);
                    shut |= bits;
                } else if (is_rename(x.tmpl)) {
                    permute(c.f, batch, U, x.tmpl);
                    std::vector<int> src((size_t)c.D);
                    for (int e = 0; e < c.D; ++e) src[(size_t)e] = c.src[(size_t)rename_source(x.tmpl, U, e)];
                    c.src.swap(src);
                } else {
                    times_diagonal(c.f, batch, U, x, pool.data());
                    each = each || x.stride;
                }
            }
            if (!ok) continue;
            const int64_t members = each ? batch : 1;
            std::vector<Mat4> mine, next;
            bool any = false;
            for (int64_t b = 0; b < members; ++b) {
                const Pool now{pool.data(), low.data(), own};
                Mat4 m = matrix_of(t, now, b), x = matrix_of(n, now, b);
                Pair s;
                const int way = passes(c, b, U, n.pos[0], n.pos[1]);
                if (way && outer_inverse(m, largest(m), &s) && is_rotation(s) && s.c.v != 0.0) {
                    any = true;
                    const Two k = s.a * s.a + s.b * s.b;
                    Mat4 in = m, turned = x;
                    for (int q = 0; q < 4; ++q) {
                        in.a[X][q] = s.a * m.a[X][q] + s.b * m.a[Y][q];
                        in.a[Y][q] = q == Z ? Two() : s.c * m.a[X][q] + s.d * m.a[Y][q];
                    }
                    // the rotation taken out, [[a, -b], [b, a]] / k by rows, or the other way round
                    const Two ga = s.a / k, gb = (way > 0 ? s.b : -s.b) / k;
                    for (int q = 1; q < 4; ++q) {
                        turned.a[q][X] = x.a[q][X] * ga + x.a[q][Y] * gb;
                        turned.a[q][Y] = x.a[q][Y] * ga - x.a[q][X] * gb;
                    }
                    m = in, x = turned;
                }
                mine.push_back(m);
                next.push_back(x);
            }
            if (!form.at_least(any)) continue;
            auto put = [&](TileOp& op, const std::vector<Mat4>& ms) {
                op.data = (int64_t)pool.size() / 2;
                op.stride = members > 1 ? 16 : 0;
                int entries = 0;
                for (const Mat4& m : ms)
                    for (int e = 0; e < 16; ++e) {
                        const Two y = tidy(m.a[e / 4][e % 4]);
                        if (e >= 4 && y.v != 0.0) entries |= 1 << (e - 4);
                        pool.push_back(y.v);
                        pool.push_back(0.0);
                        low.push_back(y.e);
                        low.push_back(0.0);
                    }
                op.zmask = ~form.at_least(entries) & ((1 << 12) - 1);
            };
            put(t, mine);
            put(n, next);
        }
}

bool lower_transfer_block(const Plan& plan, const PassDesc& pd, const BlockDesc& blk, int64_t batch, const Pool& pool,
                          Choices& form, std::vector<TransferItem>* items, int64_t* members_out) {
    const int U = blk.u, D = 1 << U;
    const int first = pd.first_op + blk.first, last = first + blk.nops;
    int64_t members = 1;
    int found = 0;
    for (int o = first; o < last; ++o) {
        if (plan.ops[(size_t)o].stride) members = batch;
        found += is_transfer(plan.ops[(size_t)o]);
    }
    if (!found) return false;
    items->clear();
    *members_out = members;
    const double overhead = 0.05;  // multiply-adds per coefficient, for an operator's own instructions
    double before = 0.0, after = 0.0;
    std::vector<Two> pend((size_t)(members * D), 1.0);  // the diagonal not yet emitted
    std::vector<std::vector<Two>> diagonals;            // the emitted ones, rounded at the end
    unsigned dep = 0, touched = 0;                         // its positions; those changed since the last one emitted
    int open = -1;
    auto emit = [&] {
        open = (int)items->size();
        items->push_back(TransferItem());
        diagonals.push_back(pend);
        std::fill(pend.begin(), pend.end(), Two(1.0));
        dep = touched = 0;
        after += 1.0 + overhead;
    };
    std::vector<char> done((size_t)blk.nops, 0);
    for (int o = first; o < last; ++o) {
        const TileOp& t = plan.ops[(size_t)o];
        const unsigned bits = positions(t);
        if (done[(size_t)(o - first)]) continue;
        if (is_diagonal(t)) {
            times_diagonal(pend, members, U, t, pool.data);
            dep |= bits | (1u << 8);  // (a factor depends on no position, and is still to be applied)
            before += 1.0 + overhead;
            continue;
        }
        if (!is_transfer(t)) {
            if (is_rename(t.tmpl)) {
                permute(pend, members, U, t.tmpl);
                if (dep & bits) dep |= bits;
            } else if (dep & bits) {
                emit();
            }
            TransferItem it;
            it.op = o;
            items->push_back(std::move(it));
            touched |= bits;
            continue;
        }
        std::vector<Mat4> m;
        for (int64_t b = 0; b < members; ++b) m.push_back(matrix_of(t, pool, b));
        before += 2.5 + overhead;
        // the next ones on the same positions, with nothing between
        for (int n = o + 1; n < last; ++n) {
            const TileOp& x = plan.ops[(size_t)n];
            if (!(positions(x) & bits)) continue;
            if (!is_transfer(x) || x.tmpl != t.tmpl) break;
            for (int64_t b = 0; b < members; ++b) m[(size_t)b] = mul(matrix_of(x, pool, b), m[(size_t)b]);
            done[(size_t)(n - first)] = 1;
            before += 2.5 + overhead;
        }
        // scales go into a diagonal before it, where there is one, else into what follows
        if (dep & (bits | (1u << 8))) emit();
        const bool left = open < 0 || (touched & bits);
        TransferItem it;
        it.pos[0] = t.pos[0], it.pos[1] = t.pos[1];
        it.mask = 0;
        const int B0 = 1 << (U - 1 - t.pos[0]), B1 = 1 << (U - 1 - t.pos[1]);
        std::vector<Two>& scales = left ? pend : diagonals.back();
        for (int64_t b = 0; b < members; ++b) {
            const Factors f = factor(m[(size_t)b], left);
            it.mask |= f.parts;
            it.v.insert(it.v.end(), {(double)f.parts, 0.0, f.v[0], f.v[1], f.w[0], f.w[1], f.s[0], f.s[1], f.shift[0], f.shift[1]});
            for (int e = 4; e < 16; ++e) it.v.push_back(f.parts & kTrDense ? m[(size_t)b].a[e / 4][e % 4].value() : 0.0);
            it.v[it.v.size() - 21] = f.shift[2];
            for (int e = 0; e < D; ++e) {
                Two& x = scales[(size_t)(b * D + e)];
                x = x * f.scale[(e & B0 ? 2 : 0) + (e & B1 ? 1 : 0)];
            }
        }
        it.mask = form.at_least(it.mask);
        items->push_back(std::move(it));
        touched |= bits;
        if (left) dep |= bits;
        after += 1.75 + overhead;
    }
    if (dep) emit();
    size_t n = 0;
    for (TransferItem& it : *items)
        if (it.op < 0 && it.mask < 0) {
            for (const Two& x : diagonals[n]) it.v.push_back(x.value());
            ++n;
        }
    return after < before && (int)items->size() <= blk.nops;
}

}  // namespace lsg
