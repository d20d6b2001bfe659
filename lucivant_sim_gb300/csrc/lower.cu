// Lowering of complex register blocks to rounds.
//
// A 2x2 unitary applied to a pair of amplitudes as it stands costs 8 multiply-adds per amplitude
// (a complex product is four real ones). Written as phases around a real plane rotation,
//   U = P * s * [[1, -t], [t, 1]] * diag(1, e)   or   P * s * [[t, -1], [1, t]] * diag(1, e),
// it costs 2: the rotation is one multiply-add per real component, because its cosine is taken out
// as a factor, and every diagonal next to it (e, s, P, diagonal gates) merges over the whole
// block into one multiplication by a table of 2^u entries (4 multiply-adds per amplitude, shared
// by all rotations of the round). Leaving the cosine out loses nothing: a0 - t * a1 is one fused
// multiply-add, its error is relative to the result, and t <= 1 (the larger of cosine and sine
// is the one taken out, `flip` says which), so the four rotations of a round grow an amplitude
// by at most 4, which the diagonal's factor has taken back before. complex64 rounds
// keep the cosine in the rotation (tile.cuh rb_round).
//
// The outer factor P need not stay in the block: a qubit that controls a cx (or meets a diagonal)
// passes a phase through it, and a cx's target passes a rotation about X, so P is taken as whichever
// the qubit's next operators let through and multiplied into the next one-bit operator on that
// qubit, in FP64 on the host. A brickwork layer then costs one diagonal per block, and no diagonal
// is left over behind it.
//
// Everything here is decided per member from that member's own data, or from the operators'
// structure alone, so a member of a batch gets the arithmetic it would get by itself: a diagonal
// that some members do not need multiplies them by exact ones.
#include <algorithm>
#include <cmath>

#include "../../include/lsg.h"
#include "lower.cuh"

namespace lsg {

namespace {

using cd = std::complex<double>;

// How far an operator may be from a rotation between phases, relative to its largest entry: gate
// matrices (and products of a few) are unitary to a few units in the last place. Anything less
// unitary stays dense.
constexpr double kUnitary = 2e-15;
// A phase this close to one is the rounding of one (gate matrices are products of a few rounded
// factors): taken as one, so the diagonal that would hold it is left out.
constexpr double kResidue = 1e-15;

struct Mat {
    cd a, b, c, d;  // rows (a, b), (c, d)
};

Mat mul(const Mat& x, const Mat& y) {
    return Mat{x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d};
}

// 1 / sqrt(x + y * y + z * z) with the rounding of the result beside it (one Newton step on the exact
// residual).
struct Exact {
    double v, err;
};
Exact inverse_length(double x, double y, double z) {
    const double yy = y * y, ye = std::fma(y, y, -yy), zz = z * z, ze = std::fma(z, z, -zz);
    const double a = x + yy, at = a - x, ae = (x - (a - at)) + (yy - at);
    const double h = a + zz, ht = h - a, he = (a - (h - ht)) + (zz - ht) + ae + ye + ze;
    const double r = 1.0 / std::sqrt(h);
    const double q = r * r, qe = std::fma(r, r, -q);
    return Exact{r, 0.5 * r * (std::fma(-h, q, 1.0) - h * qe - he * q)};
}

// s * R * diag(1, e), R = [[1, -t], [t, 1]] or, with flip, [[t, -1], [1, t]]
struct Rotation {
    cd s, s_err{0.0}, e;
    double t = 0.0, sine = 0.0;
    bool flip = false;
};

// m as a rotation; false when its first column has no real ratio or it is not that to rounding.
bool rotation(const Mat& m, Rotation* out) {
    const double p = std::abs(m.a), q = std::abs(m.c);
    const double big = std::max(p, q);
    if (!(big > 0.0) || !std::isfinite(big)) return false;
    out->flip = q > p;
    cd r, miss;
    if (!out->flip) {
        r = m.c / m.a;
        out->s = m.a;
        out->e = m.d / m.a;
        miss = m.b + r.real() * out->e * m.a;
    } else {
        r = m.a / m.c;
        out->s = m.c;
        out->e = -m.b / m.c;
        miss = m.d - r.real() * out->e * m.c;
    }
    out->t = r.real();
    if (!(std::abs(r.imag()) <= kUnitary) || !(std::abs(miss) <= kUnitary * big)) return false;
    if (!(std::abs(std::abs(out->e) - 1.0) <= 1e-9)) return false;
    // A unitary's factor s has modulus 1 / sqrt(1 + t^2): set to it beyond double precision. (Its own
    // rounding is common to all amplitudes and the norm would drift by it: 1.6e-15 over 20 layers of
    // 12 qubits, 4e-16 with it set.)
    if (std::abs(std::norm(out->s) * (1.0 + out->t * out->t) - 1.0) <= 2.0 * kUnitary) {
        const Exact u = inverse_length(0.0, out->s.real(), out->s.imag()), w = inverse_length(1.0, out->t, 0.0);
        const double k = u.v * w.v, ke = std::fma(u.v, w.v, -k) + u.v * w.err + u.err * w.v;
        const double re = out->s.real() * k, im = out->s.imag() * k;
        out->s_err = cd(std::fma(out->s.real(), k, -re) + out->s.real() * ke, std::fma(out->s.imag(), k, -im) + out->s.imag() * ke);
        out->s = cd(re, im);
    }
    if (std::abs(out->e - 1.0) < kResidue) out->e = 1.0;
    return true;
}

// The phase ph of m = diag(1, ph) * N with N's first column in a real, positive ratio.
cd outer_phase(const Mat& m) {
    if (m.a == 0.0 || m.c == 0.0) return 1.0;
    cd ph = m.c * std::conj(m.a);
    ph /= std::abs(ph);
    return std::abs(ph - 1.0) < kResidue ? cd(1.0) : ph;
}

// (divided by the phase as it is, not multiplied by its conjugate: its modulus is one only to
// rounding, and P * N is m whatever it is)
Mat without_phase(const Mat& m, cd ph) {
    return ph == cd(1.0) ? m : Mat{m.a, m.b, m.c / ph, m.d / ph};
}

// The angle of m = Rx(angle) * N with N's first column in a real ratio, its first entry the larger:
// Rx turns (y, z) of the column's Bloch vector, so that it ends at y = 0, z >= 0.
Mat outer_x(const Mat& m) {
    const double y = 2.0 * (std::conj(m.a) * m.c).imag(), z = std::norm(m.a) - std::norm(m.c);
    const double angle = (y == 0.0 && z >= 0.0) ? 0.0 : std::atan2(-y, z);
    const double c = std::cos(0.5 * angle), s = std::sin(0.5 * angle);
    return Mat{cd(c), cd(0.0, -s), cd(0.0, -s), cd(c)};
}

bool is_dense1(const TileOp& t) {
    return t.kind == LSG_OP_MATRIX && t.k == 1 && t.tmpl >= kT_DENSE1 && t.tmpl < kT_DENSE1 + 4;
}
bool is_rename(int code) { return code >= kT_X1 && code < kT_SWAP + 16; }

Mat matrix_of(const TileOp& t, const double* pool, int64_t b) {
    const double* p = pool + 2 * (t.data + (t.stride ? b * t.stride : 0));
    return Mat{cd(p[0], p[1]), cd(p[2], p[3]), cd(p[4], p[5]), cd(p[6], p[7])};
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

// A product of complex factors with the rounding errors of its steps beside it: a round's factor is
// common to all amplitudes, so its errors would add up over the program.
struct Factor {
    cd v{1.0}, err{0.0};
    void times(cd x, cd x_err) {
        auto prod = [](double a, double b, double* e) {
            const double p = a * b;
            *e = std::fma(a, b, -p);
            return p;
        };
        auto sum = [](double a, double b, double* e) {
            const double s = a + b, t = s - a;
            *e = (a - (s - t)) + (b - t);
            return s;
        };
        double e1, e2, e3, e4, e5, e6;
        const double re = sum(prod(v.real(), x.real(), &e1), -prod(v.imag(), x.imag(), &e2), &e3);
        const double im = sum(prod(v.real(), x.imag(), &e4), prod(v.imag(), x.real(), &e5), &e6);
        err = err * x + v * x_err + cd(e1 - e2 + e3, e4 + e5 + e6);
        v = cd(re, im);
    }
    cd value() const { return v + err; }
};

// A diagonal over a block's amplitudes, per member, and the positions it depends on by structure.
constexpr unsigned kNoBit = 1u << 8;
struct Diagonal {
    int64_t members;
    int D;
    std::vector<cd> v;
    unsigned dep = 0;
    Diagonal(int64_t m, int d) : members(m), D(d), v((size_t)(m * d), cd(1.0)) {}
    bool one(int64_t b) const {
        return std::all_of(v.begin() + b * D, v.begin() + (b + 1) * D, [](cd x) { return x == cd(1.0); });
    }
    bool one() const {
        return std::all_of(v.begin(), v.end(), [](cd x) { return x == cd(1.0); });
    }
    void scale(int64_t b, cd s) {
        for (int e = 0; e < D; ++e) v[(size_t)(b * D + e)] *= s;
    }
};

}  // namespace

std::vector<char> move_outer_factors(Plan& plan, int64_t batch, std::vector<double>& pool) {
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
    for (const std::vector<Touch>& seq : at) {
        std::vector<Mat> carry;  // what the operator before handed on: empty, one entry or one per member
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
            std::vector<Mat> m((size_t)members), inner, outer;
            for (int64_t b = 0; b < members; ++b) {
                m[(size_t)b] = matrix_of(t, pool.data(), b);
                if (!carry.empty()) m[(size_t)b] = mul(m[(size_t)b], carry[carry.size() == 1 ? 0 : (size_t)b]);
            }
            for (int64_t b = 0; b < members && through; ++b) {
                Rotation r;
                Mat n, p;
                if (through & 1) {
                    const cd ph = outer_phase(m[(size_t)b]);
                    n = without_phase(m[(size_t)b], ph);
                    p = Mat{cd(1.0), cd(0.0), cd(0.0), ph};
                } else {
                    p = outer_x(m[(size_t)b]);
                    const double d = p.a.real() * p.a.real() + p.b.imag() * p.b.imag();  // its determinant
                    n = mul(Mat{p.a / d, -p.b / d, -p.c / d, p.d / d}, m[(size_t)b]);
                }
                if (!rotation(n, &r)) through = 0;
                inner.push_back(n);
                outer.push_back(p);
            }
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
                for (const cd& v : {x.a, x.b, x.c, x.d}) {
                    pool.push_back(v.real());
                    pool.push_back(v.imag());
                }
        }
    }
    return moved;
}

bool lower_block(const Plan& plan, const PassDesc& pd, const BlockDesc& blk, const std::vector<char>& moved,
                 int64_t batch, const double* pool, double overhead, bool whole, LoweredBlock* out) {
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
    std::vector<Factor> gain((size_t)members);  // the open round's factors taken out
    int rounds = 0, rotations = 0;
    double cost = 0.0;

    auto emit_diag = [&](Diagonal& d) {
        LoweredItem it;
        it.code = kT_ROUND;  // without rotations
        it.mask = 16;
        it.diag = d.v;
        out->items.push_back(std::move(it));
        touched |= d.dep;
        cost += 1.0 + overhead;
        std::fill(d.v.begin(), d.v.end(), cd(1.0));
        d.dep = 0;
    };
    // The open round is complete: its factor goes into its own diagonal where a member has one, else
    // into the diagonal after it (at the block's end, when there is none either, into its own).
    auto close = [&](bool at_end) {
        if (open < 0) return;
        for (int64_t b = 0; b < members; ++b) {
            if (!pre.one(b) || (at_end && pend.one(b))) pre.scale(b, gain[(size_t)b].value());
            else pend.scale(b, gain[(size_t)b].value());
        }
        LoweredItem& it = out->items[(size_t)open];
        it.mask = (int)in_round;
        if (!pre.one()) {
            it.mask |= 16;
            it.diag = pre.v;
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
        std::vector<cd> v(pend.v.size());
        for (int64_t b = 0; b < members; ++b)
            for (int e = 0; e < D; ++e) v[(size_t)(b * D + e)] = pend.v[(size_t)(b * D + src(e))];
        pend.v.swap(v);
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
            std::vector<Rotation> r((size_t)members);
            std::vector<cd> post((size_t)members, cd(1.0));
            bool ok = true;
            for (int64_t b = 0; b < members && ok; ++b) {
                Mat m = matrix_of(t, pool, b);
                if (!moved[(size_t)o]) {
                    post[(size_t)b] = outer_phase(m);
                    m = without_phase(m, post[(size_t)b]);
                }
                ok = rotation(m, &r[(size_t)b]);
            }
            if (ok && whole)  // the rotation with its cosine and sine; what is left of s is a phase
                for (int64_t b = 0; b < members; ++b) {
                    Rotation& x = r[(size_t)b];
                    const double h = std::hypot(1.0, x.t);
                    const double c = (x.flip ? x.t : 1.0) / h, sn = (x.flip ? 1.0 : x.t) / h;
                    x.t = c;
                    x.sine = sn;
                    // the FP32 pair's length is not one to rounding, the same for every amplitude: a
                    // drift of the norm that the diagonal can take back
                    x.s *= h / std::hypot((double)(float)c, (double)(float)sn);
                    x.s_err = 0.0;
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
                    std::fill(pend.v.begin(), pend.v.end(), cd(1.0));
                    pend.dep = 0;
                    in_round = touched = 0;
                    std::fill(gain.begin(), gain.end(), Factor());
                    ++rounds;
                    cost += 1.0 + overhead;
                }
                LoweredItem& it = out->items[(size_t)open];
                for (int64_t b = 0; b < members; ++b) {
                    const Rotation& x = r[(size_t)b];
                    it.t[(size_t)(b * U + P)] = x.t;
                    it.second[(size_t)(b * U + P)] = whole ? x.sine : x.flip;
                    gain[(size_t)b].times(x.s, x.s_err);
                    for (int e = 0; e < D; ++e)
                        if (e & bit(P)) {
                            if (x.e != cd(1.0)) pre.v[(size_t)(b * D + e)] *= x.e;
                            if (post[(size_t)b] != cd(1.0)) pend.v[(size_t)(b * D + e)] *= post[(size_t)b];
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
                const double* p = pool + 2 * (t.data + (t.stride ? b * t.stride : 0));
                for (int e = 0; e < D; ++e) {
                    int j = 0;
                    for (int i = 0; i < t.k; ++i) j = (j << 1) | ((e & bit(t.pos[i])) ? 1 : 0);
                    pend.v[(size_t)(b * D + e)] *= cd(p[2 * j], p[2 * j + 1]);
                }
            }
            pend.dep |= bits | kNoBit;  // (a factor depends on no position, and is still to be applied)
            continue;
        }
        const int code = is_rename(t.tmpl) ? t.tmpl : rename_of(t, pool, members);
        if (code >= 0) {  // a rename, and its phases as a diagonal after it
            permute(code);
            if (pend.dep & bits) pend.dep |= bits;
            if (code != t.tmpl) {
                for (int64_t b = 0; b < members; ++b) {
                    const double* p = pool + 2 * (t.data + (t.stride ? b * t.stride : 0));
                    for (int e = 0; e < D; ++e) {
                        int j = 0;
                        for (int i = 0; i < t.k; ++i) j = (j << 1) | ((e & bit(t.pos[i])) ? 1 : 0);
                        pend.v[(size_t)(b * D + e)] *= cd(p[2 * j], p[2 * j + 1]);
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
    // data), emitted when some member's is not one.
    const bool left = pend.dep != 0;
    const int items = (int)out->items.size() + left;
    out->cost = cost + (left ? 1.0 + overhead : 0.0);
    if (!pend.one()) emit_diag(pend);
    return rotations > 0 && items <= blk.nops;
}

}  // namespace lsg
