// Lowering of complex register blocks to rounds.
//
// A 2x2 unitary applied to a pair of amplitudes as it stands costs 8 multiply-adds per amplitude
// (a complex product is four real ones). Written as phases around a real plane rotation,
//   U = P * s * [[1, -t], [t, 1]] * diag(1, e)   or   P * s * [[t, -1], [1, t]] * diag(1, e),
// it costs 2: the rotation is one multiply-add per real component, because its cosine is taken out
// as a factor, and every diagonal next to it (e, s, P, diagonal gates) merges over the whole
// block into one multiplication by a table of 2^u entries (4 multiply-adds per amplitude, shared
// by all rotations of the round). The cosine left out costs no accuracy in the arithmetic:
// a0 - t * a1 is one fused multiply-add, its error is relative to the result, and t <= 1 (the larger
// of cosine and sine is the one taken out, `flip` says which), so the four rotations of a round grow
// an amplitude by at most 4, which the diagonal's factor has taken back before. complex64 rounds
// keep the cosine in the rotation (tile.cuh rb_round).
//
// The outer factor P need not stay in the block: a qubit that controls a cx (or meets a diagonal)
// passes a phase through it, and a cx's target passes a rotation about X, so P is taken as whichever
// the qubit's next operators let through and multiplied into the next one-bit operator on that
// qubit, on the host. A brickwork layer then costs one diagonal per block, and no diagonal
// is left over behind it.
//
// A member of a batch gets the arithmetic it would get by itself: what is decided from values is decided
// per member from its own (a diagonal that some members do not need multiplies them by exact ones),
// all else from the operators' structure. Two decisions are taken for all members: an operator that
// is not unitary for one of them stays dense for all, and a permutation is a rename where it is the
// same one for all. The gates of circuits are unitary, and their permutations shared; beside a member
// of a caller's own list that is otherwise, a member differs by rounding from what it would be alone.
#include <algorithm>
#include <cmath>

#include "../../include/lsg.h"
#include "lower.cuh"
#include "two.cuh"

namespace lsg {

namespace {

using cd = std::complex<double>;

// How far an operator may be from a rotation between phases, relative to its largest entry. Gate
// matrices are unitary to a few units in the last place, products of n of them to some sqrt(n) times
// 1e-16: this holds for runs of some 10,000 gates on a qubit, so that whether an operator is lowered
// depends on what it is and not on a member's rounding (2e-15 left a tenth of the products of 50 gates
// dense, for every member of the batch). Anything less unitary, a matrix known to fewer digits among
// it, stays dense and is applied as given.
constexpr double kUnitary = 3e-14;
// A phase this close to one is the rounding of one (gate matrices are products of a few rounded
// factors): taken as one, so the diagonal that would hold it is left out.
constexpr double kResidue = 1e-15;

struct Cpx {
    Two re, im;
    Cpx() = default;
    Cpx(double x) : re(x) {}
    Cpx(Two x, Two y) : re(x), im(y) {}
    cd value() const { return cd(re.value(), im.value()); }
    bool one() const { return re.v + re.e == 1.0 && im.v + im.e == 0.0; }
};
LSG_INLINE Cpx conj(Cpx a) { return Cpx(a.re, -a.im); }
LSG_INLINE Cpx operator-(Cpx a) { return Cpx(-a.re, -a.im); }
LSG_INLINE Cpx operator+(Cpx a, Cpx b) { return Cpx(a.re + b.re, a.im + b.im); }
LSG_INLINE Cpx operator*(Cpx a, Cpx b) { return Cpx(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re); }
LSG_INLINE Cpx operator*(Cpx a, Two b) { return Cpx(a.re * b, a.im * b); }
LSG_INLINE Cpx operator/(Cpx a, Two b) { return a * (Two(1.0) / b); }
LSG_INLINE Two norm(Cpx a) { return a.re * a.re + a.im * a.im; }
LSG_INLINE bool zero(Cpx a) { return a.re.v == 0.0 && a.im.v == 0.0; }
// a phase, exactly one where it is the rounding of one
LSG_INLINE Cpx settled(Cpx a) {
    const double x = a.re.v - 1.0, y = a.im.v;
    return x * x + y * y < kResidue * kResidue ? Cpx(1.0) : a;
}

struct Mat {
    Cpx a, b, c, d;  // rows (a, b), (c, d)
};

Mat mul(const Mat& x, const Mat& y) {
    return Mat{x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d};
}

// The matrix nearest to m whose columns are orthogonal, [[a, -w * conj(c)], [c, w * conj(a)]]: what m is
// away from it is the rounding of its entries. (The columns keep their lengths and phases, six of m's
// eight real numbers. The nearest unitary matrix keeps four: 1.6e-15 against the gates as given,
// 2.7e-15 against those the angles stand for.) False when m is farther than rounding.
struct Unitary {
    Cpx a, c, w;
};
bool nearest(const Mat& m, Unitary* out) {
    const Two all = norm(m.a) + norm(m.b) + norm(m.c) + norm(m.d);
    if (!(all.v > 0.0) || !std::isfinite(all.v)) return false;
    const Cpx lean = (conj(m.a) * m.b + conj(m.c) * m.d) / all;  // the columns' product, over twice their length
    if (!(std::fabs(lean.re.v) + std::fabs(lean.im.v) <= kUnitary)) return false;
    out->a = m.a + -(m.b * conj(lean));
    out->c = m.c + -(m.d * conj(lean));
    out->w = (m.a * m.d + -(m.b * m.c)) / (norm(out->a) + norm(out->c));
    return std::fabs(norm(out->w).v - 1.0) <= 2.0 * kUnitary;
}

Mat matrix(const Unitary& u) { return Mat{u.a, -(u.w * conj(u.c)), u.c, u.w * conj(u.a)}; }

// The phase ph of u = diag(1, ph) * N with N's first column in a real ratio. Of its two signs, one where it
// is real (a gate without phases, h), else the one that leaves N's e (Rotation) the positive real part:
// whether a rotation needs a diagonal then does not depend on the sign of its cosine or sine.
Cpx outer_phase(const Unitary& u) {
    if (zero(u.a) || zero(u.c)) return 1.0;
    Cpx ph = u.c * conj(u.a);
    ph = ph / root(norm(ph));
    if (settled(ph).one() || settled(-ph).one()) return 1.0;
    const cd a = u.a.value(), c = u.c.value(), w = u.w.value(), p = ph.value();
    const cd e = std::norm(c) > std::norm(a) ? w * p * std::conj(c * c) : w * std::conj(p * a * a);
    return e.real() < 0.0 ? -ph : ph;
}
Unitary without_phase(const Unitary& u, Cpx ph) {
    return ph.one() ? u : Unitary{u.a, u.c * conj(ph), u.w * conj(ph)};
}

// s * R * diag(1, e), R = [[1, -t], [t, 1]] or, with flip, [[t, -1], [1, t]]
struct Rotation {
    Cpx s, e;
    Two t;
    double sine = 0.0;
    bool flip = false;
};

// m, its columns orthogonal, as a rotation; false when its first column has no real ratio.
bool rotation(const Mat& m, Rotation* out) {
    const Two aa = norm(m.a), cc = norm(m.c);
    out->flip = cc.v > aa.v;
    const Cpx top = out->flip ? m.c : m.a, rest = out->flip ? m.a : m.c;
    const Cpx back = conj(top) / (out->flip ? cc : aa);  // 1 / top
    const Cpx ratio = rest * back;
    if (!(std::fabs(ratio.im.v) <= kUnitary) || !std::isfinite(ratio.re.v)) return false;
    out->t = tidy(ratio.re);
    // (the rotation as it will be, with the rounded t, has another length)
    out->s = top * Two(1.0, out->t.v * out->t.e / (1.0 + out->t.v * out->t.v));
    out->e = settled((out->flip ? -m.b : m.d) * back);
    return true;
}

// u = Rx * N with N's first column in a real ratio, its first entry the larger: Rx turns (y, z) of the
// column's Bloch vector, so that it ends at y = 0, z >= 0. Returns N, Rx in *outer.
Unitary without_x(const Unitary& u, Mat* outer) {
    const Two y = (conj(u.a) * u.c).im * Two(2.0), z = norm(u.a) - norm(u.c);
    const double angle = (y.v == 0.0 && z.v >= 0.0) ? 0.0 : std::atan2(-y.v, z.v);
    Two co = std::cos(0.5 * angle), si = std::sin(0.5 * angle);
    // the angle's own rounding: what its sine and cosine leave of y, a turn of the half angle
    const Two s = si * co * Two(2.0), c = co * co - si * si, left = y * c + z * s, len = root(y * y + z * z);
    if (len.v > 0.0) {
        const Two turn = left / len * Two(-0.5), before = co;
        co = co - si * turn, si = si + before * turn;
    }
    const Two unit = Two(1.0) / root(co * co + si * si);
    const Cpx x(co * unit, Two()), i(Two(), si * unit);
    *outer = Mat{x, -i, -i, x};
    return Unitary{x * u.a + i * u.c, i * u.a + x * u.c, u.w};
}

bool is_dense1(const TileOp& t) {
    return t.kind == LSG_OP_MATRIX && t.k == 1 && t.tmpl >= kT_DENSE1 && t.tmpl < kT_DENSE1 + 4;
}
bool is_rename(int code) { return code >= kT_X1 && code < kT_SWAP + 16; }

// (entries that move_outer_factors appended have their rounding errors in `low`)
Mat matrix_of(const TileOp& t, const Pool& pool, int64_t b) {
    const int64_t at = 2 * (t.data + (t.stride ? b * t.stride : 0));
    const double* p = pool.data + at;
    if (at < pool.own) return Mat{Cpx(p[0], p[1]), Cpx(p[2], p[3]), Cpx(p[4], p[5]), Cpx(p[6], p[7])};
    const double* e = pool.low + (at - pool.own);
    auto entry = [&](int i) { return Cpx(Two(p[i], e[i]), Two(p[i + 1], e[i + 1])); };
    return Mat{entry(0), entry(2), entry(4), entry(6)};
}

// What an operator lets through on its local bit `lb`: 1 phases, 2 rotations about X.
int lets_through(const TileOp& t, int lb) {
    if (t.kind == LSG_OP_DIAG) return 1;
    if (t.tmpl < kT_CX || t.tmpl >= kT_CX + 16) return 0;
    const int control = (t.tmpl - kT_CX) / 4;
    for (int i = 0; i < t.k; ++i)
        if (t.lb[i] == lb) return t.pos[i] == control ? 1 : 2;
    return 0;
}

// The rename code of a permutation with phases whose sources are those of an X, a cx or a swap for
// every member, or -1.
int rename_of(const TileOp& t, const double* pool, int64_t members) {
    if (t.kind != LSG_OP_PERM || t.k > 2 || t.tmpl < kT_PERM1 || t.tmpl >= kT_PERM2 + 16) return -1;
    const int d = 1 << t.k;
    int want[4] = {0, 0, 0, 0};
    for (int64_t b = 0; b < (t.stride ? members : 1); ++b)
        for (int r = 0; r < d; ++r) {
            const int src = (int)pool[2 * (t.data + (t.stride ? b * t.stride : 0) + d + r)];
            if (b && src != want[r]) return -1;
            want[r] = src;
        }
    auto is = [&](int a, int b, int c, int e) { return want[0] == a && want[1] == b && want[2] == c && want[3] == e; };
    if (t.k == 1) return want[0] == 1 && want[1] == 0 ? kT_X1 + t.pos[0] : -1;
    if (is(0, 1, 3, 2)) return kT_CX + 4 * t.pos[0] + t.pos[1];
    if (is(0, 3, 2, 1)) return kT_CX + 4 * t.pos[1] + t.pos[0];
    return is(0, 2, 1, 3) ? kT_SWAP + 4 * t.pos[0] + t.pos[1] : -1;
}

// A diagonal over a block's amplitudes, per member, and the positions it depends on by structure.
constexpr unsigned kNoBit = 1u << 8;
struct Diagonal {
    int64_t members;
    int D;
    std::vector<Cpx> v;
    unsigned dep = 0;
    Diagonal(int64_t m, int d) : members(m), D(d), v((size_t)(m * d), Cpx(1.0)) {}
    bool one(int64_t b) const {
        return std::all_of(v.begin() + b * D, v.begin() + (b + 1) * D, [](const Cpx& x) { return x.one(); });
    }
    bool one() const {
        return std::all_of(v.begin(), v.end(), [](const Cpx& x) { return x.one(); });
    }
    void scale(int64_t b, Cpx s) {
        for (int e = 0; e < D; ++e) times(b, e, s);
    }
    void times(int64_t b, int e, Cpx s) {
        Cpx& x = v[(size_t)(b * D + e)];
        x = x.one() ? s : x * s;
    }
    std::vector<cd> rounded() const {
        std::vector<cd> out(v.size());
        std::transform(v.begin(), v.end(), out.begin(), [](const Cpx& x) { return x.value(); });
        return out;
    }
};

}  // namespace

std::vector<char> move_outer_factors(Plan& plan, int64_t batch, std::vector<double>& pool, std::vector<double>& low) {
    const int64_t own = (int64_t)pool.size();
    std::vector<char> moved(plan.ops.size(), 0);
    struct Touch {
        int op, lb;
        bool block;
    };
    std::vector<Touch> at[64];  // the operators on each register bit, in execution order
    for (const PassDesc& pd : plan.passes)
        for (int bi = pd.first_block; bi < pd.first_block + pd.nblocks; ++bi) {
            const BlockDesc& blk = plan.blocks[(size_t)bi];
            for (int o = pd.first_op + blk.first; o < pd.first_op + blk.first + blk.nops; ++o) {
                const TileOp& t = plan.ops[(size_t)o];
                for (int i = 0; i < t.k; ++i)
                    at[t.lb[i] < pd.L ? t.lb[i] : pd.hi[t.lb[i] - pd.L]].push_back(Touch{o, t.lb[i], !blk.generic});
            }
        }
    std::vector<Mat> m, inner, outer;
    std::vector<Mat> carry;  // what the operator before handed on: empty, one entry or one per member
    bool phases = false;     // diag(1, phase)
    for (const std::vector<Touch>& seq : at) {
        carry.clear();
        for (size_t i = 0; i < seq.size(); ++i) {
            TileOp& t = plan.ops[(size_t)seq[i].op];
            if (!seq[i].block || !is_dense1(t)) continue;
            // what everything up to the next one-bit operator on this bit lets through
            int through = 3;
            size_t j = i + 1;
            for (; j < seq.size() && through; ++j) {
                const TileOp& n = plan.ops[(size_t)seq[j].op];
                if (seq[j].block && is_dense1(n)) break;
                through &= seq[j].block ? lets_through(n, seq[j].lb) : 0;
            }
            if (j >= seq.size()) through = 0;
            const int64_t members = std::max<int64_t>(t.stride ? batch : 1, (int64_t)carry.size());
            m.resize((size_t)members);
            inner.clear(), outer.clear();
            for (int64_t b = 0; b < members; ++b) {
                m[(size_t)b] = matrix_of(t, Pool{pool.data(), low.data(), own}, b);
                if (carry.empty()) continue;
                const Mat& c = carry[carry.size() == 1 ? 0 : (size_t)b];
                Mat& x = m[(size_t)b];
                if (!phases) x = mul(x, c);
                else if (!c.d.one()) x.b = x.b * c.d, x.d = x.d * c.d;
            }
            for (int64_t b = 0; b < members && through; ++b) {
                Unitary u;
                Mat p;
                if (!nearest(m[(size_t)b], &u)) {
                    through = 0;
                    break;
                }
                if (through & 1) {
                    const Cpx ph = outer_phase(u);
                    u = without_phase(u, ph);
                    p = Mat{Cpx(1.0), Cpx(0.0), Cpx(0.0), ph};
                } else {
                    u = without_x(u, &p);
                }
                inner.push_back(matrix(u));
                outer.push_back(p);
            }
            phases = through & 1;
            const bool carried = !carry.empty();
            carry.clear();
            if (through) {
                m.swap(inner);
                carry.swap(outer);
                moved[(size_t)seq[i].op] = 1;
            }
            if (!through && !carried) continue;
            t.data = (int64_t)pool.size() / 2;
            t.stride = members > 1 ? 4 : 0;
            for (const Mat& x : m)
                for (const Cpx& v : {x.a, x.b, x.c, x.d})
                    for (Two part : {tidy(v.re), tidy(v.im)}) {
                        pool.push_back(part.v);
                        low.push_back(part.e);
                    }
        }
    }
    return moved;
}

bool lower_block(const Plan& plan, const PassDesc& pd, const BlockDesc& blk, const std::vector<char>& moved,
                 int64_t batch, const Pool& pool, double overhead, bool whole, Choices& form, LoweredBlock* out) {
    const int U = blk.u, D = 1 << U;
    const int first = pd.first_op + blk.first, last = first + blk.nops;
    int64_t members = 1;
    for (int o = first; o < last; ++o)
        if (plan.ops[(size_t)o].stride) members = batch;
    out->items.clear();
    out->members = members;
    auto bit = [&](int P) { return 1 << (U - 1 - P); };  // block position -> bit of the group index

    Diagonal pend(members, D);  // diagonals since the open round's rotations
    int open = -1;              // the round that later rotations may still join
    unsigned in_round = 0, touched = 0;
    Diagonal pre(members, D);   // the open round's diagonal
    std::vector<Cpx> gain((size_t)members, Cpx(1.0));  // the open round's factors taken out
    std::vector<Rotation> r;
    std::vector<Cpx> post;
    int rounds = 0, rotations = 0;
    double cost = 0.0;

    auto emit_diag = [&](Diagonal& d) {
        LoweredItem it;
        it.code = kT_ROUND;  // without rotations
        it.mask = 16;
        it.diag = d.rounded();
        out->items.push_back(std::move(it));
        touched |= d.dep;
        cost += 1.0 + overhead;
        std::fill(d.v.begin(), d.v.end(), Cpx(1.0));
        d.dep = 0;
    };
    // The open round is complete: its factor goes into its own diagonal where a member has one, else
    // into the diagonal after it (at the block's end, when there is none either, into its own).
    auto close = [&](bool at_end) {
        if (open < 0) return;
        for (int64_t b = 0; b < members; ++b) {
            if (!pre.one(b) || (at_end && pend.one(b))) pre.scale(b, gain[(size_t)b]);
            else pend.scale(b, gain[(size_t)b]);
        }
        LoweredItem& it = out->items[(size_t)open];
        it.mask = (int)in_round;
        if (form.at_least(!pre.one())) {
            it.mask |= 16;
            it.diag = pre.rounded();
        }
        open = -1;
    };
    // Mixtures (a member's branch of a noise channel, nearly always the identity) wait: they commute
    // with what follows on other bits, so a block's channels share the one diagonal before them.
    std::vector<int> late;
    unsigned late_bits = 0;
    auto keep = [&](int o, int code) {
        LoweredItem it;
        it.code = kKeepOp;
        it.op = o;
        it.tmpl = code;
        out->items.push_back(std::move(it));
    };
    auto flush_late = [&] {
        if (late.empty()) return;
        if (pend.dep & late_bits) emit_diag(pend);
        for (int o : late) keep(o, plan.ops[(size_t)o].tmpl);
        touched |= late_bits;
        late.clear();
        late_bits = 0;
    };
    auto permute = [&](int code) {  // the rename moves the diagonal that stands before it
        auto src = [&](int e) {
            if (code < kT_CX) return e ^ bit(code - kT_X1);
            if (code < kT_SWAP) return (e & bit((code - kT_CX) / 4)) ? e ^ bit((code - kT_CX) % 4) : e;
            const int x = bit((code - kT_SWAP) / 4), y = bit((code - kT_SWAP) % 4);
            return ((e & x) != 0) != ((e & y) != 0) ? e ^ x ^ y : e;
        };
        if (!pend.dep) return;  // ones
        Cpx v[16];
        for (int64_t b = 0; b < members; ++b) {
            Cpx* now = pend.v.data() + b * D;
            std::copy(now, now + D, v);
            for (int e = 0; e < D; ++e) now[e] = v[src(e)];
        }
    };

    for (int o = first; o < last; ++o) {
        const TileOp& t = plan.ops[(size_t)o];
        unsigned bits = 0;
        for (int i = 0; i < t.k; ++i) bits |= 1u << t.pos[i];
        if (bits & late_bits) flush_late();
        if (t.kind == kOpMixture) {
            late.push_back(o);
            late_bits |= bits;
            cost += 0.25 + overhead;
            continue;
        }
        if (is_dense1(t)) {
            const int P = t.pos[0];
            r.assign((size_t)members, Rotation());
            post.assign((size_t)members, Cpx(1.0));
            bool ok = true;
            for (int64_t b = 0; b < members && ok; ++b) {
                Mat m = matrix_of(t, pool, b);
                if (!moved[(size_t)o]) {
                    Unitary u;
                    ok = nearest(m, &u);
                    if (!ok) break;
                    post[(size_t)b] = outer_phase(u);
                    m = matrix(without_phase(u, post[(size_t)b]));
                }
                ok = rotation(m, &r[(size_t)b]);
            }
            if (ok && whole)  // the rotation with its cosine and sine; what is left of s is a phase
                for (int64_t b = 0; b < members; ++b) {
                    Rotation& x = r[(size_t)b];
                    const double h = std::hypot(1.0, x.t.v);
                    const double c = (x.flip ? x.t.v : 1.0) / h, sn = (x.flip ? 1.0 : x.t.v) / h;
                    x.t = c;
                    x.sine = sn;
                    // the FP32 pair's length is not one to rounding, the same for every amplitude: a
                    // drift of the norm that the diagonal can take back
                    x.s = x.s * Two(h / std::hypot((double)(float)c, (double)(float)sn));
                }
            if (ok) {
                if (open < 0 || ((in_round | touched | pend.dep) & bits)) {
                    close(false);
                    LoweredItem it;
                    it.code = kT_ROUND;
                    it.t.assign((size_t)(members * U), 0.0);
                    it.second.assign((size_t)(members * U), 0.0);
                    open = (int)out->items.size();
                    out->items.push_back(std::move(it));
                    pre = pend;
                    std::fill(pend.v.begin(), pend.v.end(), Cpx(1.0));
                    pend.dep = 0;
                    in_round = touched = 0;
                    std::fill(gain.begin(), gain.end(), Cpx(1.0));
                    ++rounds;
                    cost += 1.0 + overhead;
                }
                LoweredItem& it = out->items[(size_t)open];
                for (int64_t b = 0; b < members; ++b) {
                    const Rotation& x = r[(size_t)b];
                    it.t[(size_t)(b * U + P)] = x.t.value();
                    it.second[(size_t)(b * U + P)] = whole ? x.sine : x.flip;
                    gain[(size_t)b] = gain[(size_t)b].one() ? x.s : gain[(size_t)b] * x.s;
                    for (int e = 0; e < D; ++e)
                        if (e & bit(P)) {
                            if (!x.e.one()) pre.times(b, e, x.e);
                            if (!post[(size_t)b].one()) pend.times(b, e, post[(size_t)b]);
                        }
                }
                if (!moved[(size_t)o]) pend.dep |= bits | kNoBit;
                in_round |= bits;
                ++rotations;
                cost += 0.5;
                continue;
            }
        }
        if (t.tmpl == kT_DIAG || t.tmpl == kT_SCALE) {
            for (int64_t b = 0; b < members; ++b) {
                const double* p = pool.data + 2 * (t.data + (t.stride ? b * t.stride : 0));
                for (int e = 0; e < D; ++e) {
                    int j = 0;
                    for (int i = 0; i < t.k; ++i) j = (j << 1) | ((e & bit(t.pos[i])) ? 1 : 0);
                    pend.times(b, e, Cpx(p[2 * j], p[2 * j + 1]));
                }
            }
            pend.dep |= bits | kNoBit;  // (a factor depends on no position, and is still to be applied)
            continue;
        }
        const int code = is_rename(t.tmpl) ? t.tmpl : rename_of(t, pool.data, members);
        if (code >= 0) {  // a rename, and its phases as a diagonal after it
            permute(code);
            if (pend.dep & bits) pend.dep |= bits;
            if (code != t.tmpl) {
                for (int64_t b = 0; b < members; ++b) {
                    const double* p = pool.data + 2 * (t.data + (t.stride ? b * t.stride : 0));
                    for (int e = 0; e < D; ++e) {
                        int j = 0;
                        for (int i = 0; i < t.k; ++i) j = (j << 1) | ((e & bit(t.pos[i])) ? 1 : 0);
                        pend.times(b, e, Cpx(p[2 * j], p[2 * j + 1]));
                    }
                }
                pend.dep |= bits;
            }
            cost += 0.25 + overhead;
        } else {  // any other operator: diagonals on its bits go before it
            if (pend.dep & bits) emit_diag(pend);
            cost += (t.kind == LSG_OP_PERM ? 1.0 : t.k == 1 ? 2.0 : 4.0) + overhead;
        }
        touched |= bits;
        keep(o, code >= 0 ? code : t.tmpl);
    }
    flush_late();
    close(true);
    // A diagonal left over: by structure (whether the block is lowered is the same for every member's
    // data), emitted when some member's is not one (or has not been).
    const bool left = pend.dep != 0;
    const int items = (int)out->items.size() + left;
    out->cost = cost + (left ? 1.0 + overhead : 0.0);
    if (left && form.at_least(!pend.one())) emit_diag(pend);
    return rotations > 0 && items <= blk.nops;
}

}  // namespace lsg
