// Host planner: classify circuit gates and fuse them into tile passes.
//
// Classification follows the reference's dispatch (src/qfvm/simulator.hpp:
// 12-113) and matrix construction (src/qfvm/statevector.hpp:340-437); the
// fuser is this engine's own: gates are grouped into passes over tiles of T
// qubits (the low L qubits are always in the tile so that HBM accesses are
// contiguous runs), and inside a pass into register rounds of R qubits.
// Diagonal gates and controls need no tile membership: they are evaluated
// from each amplitude's global index, so only the targets of non-diagonal
// gates constrain the schedule.
#include <algorithm>
#include <cmath>
#include <complex>
#include <climits>
#include <cstring>
#include <list>
#include <mutex>
#include <set>
#include <string>

#include "engine.h"

namespace qsv {

int amp_bytes(int precision) { return precision == QFVM_C64 ? 8 : 16; }

// Largest state handled by the whole-state (single CTA, shared memory) kernel.
int small_max_qubits(int precision) { return precision == QFVM_C64 ? 14 : 13; }

// Built-in shapes (the autotuner's choices on GB300 for the random-layer and
// hardware-efficient workloads; a tuned table entry overrides them).
void default_shape(int n, int precision, int* T, int* R) {
    if (precision == QFVM_C64) {
        *T = 13;
        *R = 5;
    } else if (precision == QFVM_C128_DS) {
        *T = 12;
        *R = 3;
    } else {
        *T = 11;
        *R = 4;
    }
    (void)n;
}

namespace {

using cd = std::complex<double>;

void set_diag(GOp& g, cd d0, cd d1) {
    g.kind = K_DIAG;
    g.coef = {d0.real(), d0.imag(), d1.real(), d1.imag()};
    if (d0 == cd(1.0, 0.0)) {
        g.flags |= F_D0_ONE;
        if (d1 == cd(-1.0, 0.0)) {
            g.flags |= F_D1_SPEC;
            g.special = SP_NEG1;
        } else if (d1 == cd(0.0, 1.0)) {
            g.flags |= F_D1_SPEC;
            g.special = SP_I;
        } else if (d1 == cd(0.0, -1.0)) {
            g.flags |= F_D1_SPEC;
            g.special = SP_NEGI;
        }
    }
}

bool is_zero(cd z) { return z.real() == 0.0 && z.imag() == 0.0; }

}  // namespace

bool classify(int n, const qfvm_op* ops, int64_t n_ops, const double* matpool, int64_t matpool_len,
              std::vector<GOp>* out, std::string* err) {
    out->clear();
    out->reserve(static_cast<size_t>(n_ops));
    const double PI_ = 3.14159265358979323846;
    for (int64_t i = 0; i < n_ops; ++i) {
        const qfvm_op& o = ops[i];
        const int nq = o.nqubits;
        if (nq < 1 || nq > QFVM_MAX_OP_QUBITS) {
            *err = "op " + std::to_string(i) + ": bad qubit count " + std::to_string(nq);
            return false;
        }
        uint64_t seen = 0;
        for (int j = 0; j < nq; ++j) {
            int q = o.qubits[j];
            if (q < 0 || q >= n) {
                *err = "op " + std::to_string(i) + ": qubit " + std::to_string(q) + " outside a " +
                       std::to_string(n) + "-qubit state";
                return false;
            }
            if (seen & (1ULL << q)) {
                *err = "op " + std::to_string(i) + ": repeated qubit " + std::to_string(q);
                return false;
            }
            seen |= 1ULL << q;
        }
        for (int j = 0; j < 4; ++j) {
            if (!std::isfinite(o.params[j])) {
                *err = "op " + std::to_string(i) + ": non-finite parameter";
                return false;
            }
        }
        GOp g;
        g.src = static_cast<int>(i);
        g.slot = o.slot;
        if (o.slot >= 0 && (o.kind == QFVM_OP_RX || o.kind == QFVM_OP_RY || o.kind == QFVM_OP_RZ ||
                            o.kind == QFVM_OP_P || o.kind == QFVM_OP_CP || o.kind == QFVM_OP_RZZ))
            g.bkind = static_cast<uint8_t>(o.kind);
        const int* q = o.qubits;
        auto need = [&](int k) {
            if (nq < k) {
                *err = "op " + std::to_string(i) + ": gate kind " + std::to_string(o.kind) + " needs " +
                       std::to_string(k) + " qubits";
                return false;
            }
            return true;
        };
        const double th = o.params[0];
        switch (o.kind) {
            case QFVM_OP_X:
                g.kind = K_X;
                g.t0 = q[0];
                break;
            case QFVM_OP_Y:
                g.kind = K_Y;
                g.t0 = q[0];
                break;
            case QFVM_OP_Z:
                g.pmask = 1ULL << q[0];
                set_diag(g, 1.0, -1.0);
                break;
            case QFVM_OP_H: {
                const double s = 1. / std::sqrt(2.);
                g.kind = K_REAL;
                g.t0 = q[0];
                g.coef = {s, s, s, -s};
                break;
            }
            case QFVM_OP_S:
                g.pmask = 1ULL << q[0];
                set_diag(g, 1.0, cd(0, 1));
                break;
            case QFVM_OP_SDG:
                g.pmask = 1ULL << q[0];
                set_diag(g, 1.0, cd(0, -1));
                break;
            case QFVM_OP_T:
            case QFVM_OP_TDG: {
                const double a = (o.kind == QFVM_OP_T ? 1.0 : -1.0) * PI_ / 4.;
                g.pmask = 1ULL << q[0];
                set_diag(g, 1.0, cd(std::cos(a), std::sin(a)));
                break;
            }
            case QFVM_OP_P:
                g.pmask = 1ULL << q[0];
                set_diag(g, 1.0, cd(std::cos(th), std::sin(th)));
                break;
            case QFVM_OP_RX:
                g.kind = K_RX;
                g.t0 = q[0];
                g.coef = {std::cos(th / 2), std::sin(th / 2)};
                break;
            case QFVM_OP_RY: {
                const double c = std::cos(th / 2), s = std::sin(th / 2);
                g.kind = K_REAL;
                g.t0 = q[0];
                g.coef = {c, -s, s, c};
                break;
            }
            case QFVM_OP_RZ: {
                const double h = th / 2.;
                g.pmask = 1ULL << q[0];
                set_diag(g, cd(std::cos(-h), std::sin(-h)), cd(std::cos(h), std::sin(h)));
                break;
            }
            case QFVM_OP_CX:
                if (!need(2)) return false;
                g.kind = K_X;
                g.cmask = 1ULL << q[0];
                g.t0 = q[1];
                break;
            case QFVM_OP_CZ:
                if (!need(2)) return false;
                g.cmask = 1ULL << q[0];
                g.pmask = 1ULL << q[1];
                set_diag(g, 1.0, -1.0);
                break;
            case QFVM_OP_CP:
                if (!need(2)) return false;
                g.cmask = 1ULL << q[0];
                g.pmask = 1ULL << q[1];
                set_diag(g, 1.0, cd(std::cos(th), std::sin(th)));
                break;
            case QFVM_OP_CCX:
                if (!need(3)) return false;
                g.kind = K_X;
                g.cmask = (1ULL << q[0]) | (1ULL << q[1]);
                g.t0 = q[2];
                break;
            case QFVM_OP_RZZ: {
                // simulator.hpp:90-94 applies cx . rz . cx: a phase by the parity of the two qubits.
                if (!need(2)) return false;
                const double h = th / 2.;
                g.pmask = (1ULL << q[0]) | (1ULL << q[1]);
                set_diag(g, cd(std::cos(-h), std::sin(-h)), cd(std::cos(h), std::sin(h)));
                break;
            }
            case QFVM_OP_MATRIX: {
                const int nc = o.ncontrols;
                const int k = nq - nc;
                if (nc < 0 || k < 1) {
                    *err = "op " + std::to_string(i) + ": matrix gate without a target";
                    return false;
                }
                if (k > MAX_DENSE_TARGETS) {
                    *err = "op " + std::to_string(i) + ": " + std::to_string(k) +
                           "-target matrix gates are not supported (at most " + std::to_string(MAX_DENSE_TARGETS) +
                           " targets)";
                    return false;
                }
                const int64_t dim = 1LL << k;
                if (o.mat_dim != dim || o.mat_offset < 0 || o.mat_offset + dim * dim > matpool_len) {
                    *err = "op " + std::to_string(i) + ": matrix does not match its target count";
                    return false;
                }
                const cd* m = reinterpret_cast<const cd*>(matpool) + o.mat_offset;
                for (int j = 0; j < nc; ++j) g.cmask |= 1ULL << q[j];
                for (int64_t j = 0; j < dim * dim; ++j) {
                    if (!std::isfinite(m[j].real()) || !std::isfinite(m[j].imag())) {
                        *err = "op " + std::to_string(i) + ": non-finite matrix entry";
                        return false;
                    }
                }
                if (k == 1) {
                    const int t = q[nc];
                    g.t0 = t;
                    if (is_zero(m[1]) && is_zero(m[2])) {
                        g.pmask = 1ULL << t;
                        set_diag(g, m[0], m[3]);
                    } else if (is_zero(m[0]) && is_zero(m[3]) && m[1] == cd(1, 0) && m[2] == cd(1, 0)) {
                        g.kind = K_X;
                    } else if (m[0].imag() == 0 && m[1].imag() == 0 && m[2].imag() == 0 && m[3].imag() == 0) {
                        g.kind = K_REAL;
                        g.coef = {m[0].real(), m[1].real(), m[2].real(), m[3].real()};
                    } else {
                        g.kind = K_DENSE;
                        g.coef.resize(8);
                        for (int j = 0; j < 4; ++j) {
                            g.coef[2 * j] = m[j].real();
                            g.coef[2 * j + 1] = m[j].imag();
                        }
                    }
                } else if (k == 2) {
                    g.t0 = q[nc];
                    g.t1 = q[nc + 1];
                    bool swap = true;
                    for (int r = 0; r < 4 && swap; ++r)
                        for (int c = 0; c < 4; ++c) {
                            int want = (r == 0 && c == 0) || (r == 3 && c == 3) || (r == 1 && c == 2) ||
                                       (r == 2 && c == 1);
                            if (m[r * 4 + c] != cd(want ? 1.0 : 0.0, 0.0)) {
                                swap = false;
                                break;
                            }
                        }
                    if (swap) {
                        g.kind = K_SWAP;
                    } else {
                        g.kind = K_DENSE2;
                        g.coef.resize(32);
                        for (int j = 0; j < 16; ++j) {
                            g.coef[2 * j] = m[j].real();
                            g.coef[2 * j + 1] = m[j].imag();
                        }
                    }
                } else if (k <= MAXK) {
                    g.kind = K_DENSEK;
                    g.k = k;
                    for (int j = 0; j < k; ++j) g.tk[j] = q[nc + j];
                    g.coef.resize(static_cast<size_t>(2 * dim * dim));
                    for (int64_t j = 0; j < dim * dim; ++j) {
                        g.coef[2 * j] = m[j].real();
                        g.coef[2 * j + 1] = m[j].imag();
                    }
                } else {
                    // wide gate: targets in ascending order, the matrix's index
                    // bits relabelled to match (a permutation of entries, exact)
                    g.kind = K_DENSEK;
                    g.k = k;
                    int ord[MAX_DENSE_TARGETS];
                    for (int j = 0; j < k; ++j) ord[j] = j;
                    std::sort(ord, ord + k, [&](int a, int b) { return q[nc + a] < q[nc + b]; });
                    for (int j = 0; j < k; ++j) g.tk[j] = q[nc + ord[j]];
                    std::vector<int64_t> old_of(static_cast<size_t>(dim));
                    for (int64_t v = 0; v < dim; ++v) {
                        int64_t o2 = 0;
                        for (int j = 0; j < k; ++j)
                            if ((v >> j) & 1) o2 |= int64_t{1} << ord[j];
                        old_of[static_cast<size_t>(v)] = o2;
                    }
                    g.coef.resize(static_cast<size_t>(2 * dim * dim));
                    for (int64_t r = 0; r < dim; ++r)
                        for (int64_t c = 0; c < dim; ++c) {
                            const cd e = m[old_of[static_cast<size_t>(r)] * dim + old_of[static_cast<size_t>(c)]];
                            g.coef[static_cast<size_t>(2 * (r * dim + c))] = e.real();
                            g.coef[static_cast<size_t>(2 * (r * dim + c) + 1)] = e.imag();
                        }
                }
                break;
            }
            default:
                *err = "op " + std::to_string(i) + ": kind " + std::to_string(o.kind) +
                       " is not a gate this entry point applies";
                return false;
        }
        if (g.kind == K_X || g.kind == K_Y || g.kind == K_REAL || g.kind == K_RX || g.kind == K_DENSE) {
            if (g.cmask & (1ULL << g.t0)) {
                *err = "op " + std::to_string(i) + ": target is also a control";
                return false;
            }
        }
        // generator of a parameterised gate: dG/dtheta = -i/2 Q G
        // (rotations exp(-i theta Q / 2); phase gates diag(1, e^{i l}) give Q = -2 proj)
        {
            const uint64_t b0 = 1ULL << q[0];
            switch (o.kind) {
                case QFVM_OP_RX: g.has_gen = true; g.gx = b0; break;
                case QFVM_OP_RY: g.has_gen = true; g.gx = b0; g.gz = b0; g.gny = 1; break;
                case QFVM_OP_RZ: g.has_gen = true; g.gz = b0; break;
                case QFVM_OP_RZZ: g.has_gen = true; g.gz = b0 | (1ULL << q[1]); break;
                case QFVM_OP_P: g.has_gen = true; g.gcmask = b0; g.gscale = -2.0; break;
                case QFVM_OP_CP: g.has_gen = true; g.gcmask = b0 | (1ULL << q[1]); g.gscale = -2.0; break;
                case QFVM_OP_MATRIX: {
                    uint64_t tm = 0, cm = 0;
                    for (int j = 0; j < o.ncontrols; ++j) cm |= 1ULL << q[j];
                    for (int j = o.ncontrols; j < nq; ++j) tm |= 1ULL << q[j];
                    const int nt = nq - o.ncontrols;
                    switch (o.gen) {
                        case QFVM_GEN_X: g.has_gen = true; g.gx = tm; g.gcmask = cm; break;
                        case QFVM_GEN_Y: g.has_gen = true; g.gx = tm; g.gz = tm; g.gny = nt; g.gcmask = cm; break;
                        case QFVM_GEN_Z: g.has_gen = true; g.gz = tm; g.gcmask = cm; break;
                        case QFVM_GEN_PHASE: g.has_gen = true; g.gcmask = tm | cm; g.gscale = -2.0; break;
                        default: break;
                    }
                    break;
                }
                default: break;
            }
        }
        out->push_back(std::move(g));
    }
    return true;
}

double gop_bytes(const GOp& g, int n, int precision) {
    const double N = std::ldexp(1.0, n);
    const int nc = __builtin_popcountll(g.cmask);
    double amps = N / std::ldexp(1.0, nc);
    switch (g.kind) {
        case K_DIAG:
            if (g.flags & F_D0_ONE) amps *= 0.5;
            break;
        case K_SWAP:
            amps *= 0.5;
            break;
        default:
            break;
    }
    return 2.0 * amp_bytes(precision) * amps;
}

namespace {

// Qubit actions for commutation: two gates commute if on every shared qubit
// both act diagonally (controls, phases) or both act as X (targets of X/CX).
enum Act : uint8_t { A_Z = 1, A_X = 2, A_G = 4 };

void gop_actions(const GOp& g, std::vector<std::pair<int, uint8_t>>* acts) {
    acts->clear();
    for (int q = 0; q < 64; ++q) {
        if (g.cmask & (1ULL << q)) acts->push_back({q, A_Z});
        if (g.pmask & (1ULL << q)) acts->push_back({q, A_Z});
    }
    switch (g.kind) {
        case K_X: acts->push_back({g.t0, A_X}); break;
        case K_DIAG: break;
        case K_SWAP:
        case K_DENSE2:
            acts->push_back({g.t0, A_G});
            acts->push_back({g.t1, A_G});
            break;
        case K_DENSEK:
            for (int j = 0; j < g.k; ++j) acts->push_back({g.tk[j], A_G});
            break;
        case K_PROBE:
            // a probe of Q commutes with a gate that commutes with Q: Z bits and
            // the projector act diagonally, pure flip bits as X, Y bits as both
            for (int q = 0; q < 64; ++q) {
                const uint64_t b = 1ULL << q;
                if (g.xmask & b) acts->push_back({q, (g.pmask & b) ? A_G : A_X});
            }
            break;
        default: acts->push_back({g.t0, A_G}); break;
    }
}

void gop_targets(const GOp& g, std::vector<int>* t) {
    t->clear();
    switch (g.kind) {
        case K_DIAG: break;
        case K_SWAP:
        case K_DENSE2:
            t->push_back(g.t0);
            t->push_back(g.t1);
            break;
        case K_DENSEK:
            for (int j = 0; j < g.k; ++j) t->push_back(g.tk[j]);
            break;
        case K_PROBE:  // flipped qubits pair amplitudes: they must be register bits
            for (int q = 0; q < 64; ++q)
                if (g.xmask & (1ULL << q)) t->push_back(q);
            break;
        default: t->push_back(g.t0); break;
    }
}

// Copy a gop's coefficients into the pool and return the offset.
uint32_t push_coef(HostPlan* p, const GOp& g) {
    // every block starts 4-aligned (the kernels read coefficients four at a
    // time with 16-byte loads); the padding stays zero
    while (p->coef.size() % 4) p->coef.push_back(0.0);
    uint32_t off = static_cast<uint32_t>(p->coef.size());
    p->coef.insert(p->coef.end(), g.coef.begin(), g.coef.end());
    if (g.bkind != 0 && g.slot >= 0 && g.kind != K_PROBE)
        p->binds.push_back(Bind{off, g.bkind, g.bsign, static_cast<uint16_t>(g.special == SP_BOUND_RZ), g.slot});
    return off;
}

// Whole-state op record: all masks over global index bits.
KOp global_kop(HostPlan* p, const GOp& g) {
    KOp k;
    std::memset(&k, 0, sizeof(k));
    k.kind = g.kind;
    k.flags = g.flags;
    k.special = g.special;
    k.t0 = static_cast<uint8_t>(g.t0 < 0 ? 0 : g.t0);
    k.t1 = static_cast<uint8_t>(g.t1 < 0 ? 0 : g.t1);
    k.k = static_cast<uint8_t>(g.k);
    for (int j = 0; j < g.k && j < MAXK; ++j) k.tk[j] = static_cast<uint8_t>(g.tk[j]);
    k.cthr = g.cmask;
    k.pthr = g.pmask;
    if (g.kind == K_DENSEK && g.k > MAXK) {
        k.pthr = 0;
        for (int j = 0; j < g.k; ++j) k.pthr |= 1ULL << g.tk[j];  // ascending targets as a mask
    }
    if (g.kind == K_PROBE) {
        k.xreg = static_cast<uint32_t>(g.xmask);  // whole-state kernels: global flip bits (n <= 14)
        k.probe = static_cast<uint16_t>(p->probe_slot.size());
        p->probe_slot.push_back(g.slot);
    }
    k.coef = push_coef(p, g);
    return k;
}

// Thread-bit order for a register round: the first lanes get positions that
// land on distinct slot bits of the tile layout (tile_slot_bit), so each
// wavefront of the round's shared-memory accesses (`access` bytes per lane)
// covers distinct bank groups.
void order_thread_bits(std::vector<int>& free_pos, int elem_bytes, int access) {
    const int nslot = access == 16 ? 3 : 4;  // 128 / access = 2^nslot slots per wavefront
    std::vector<int> head, rest;
    std::vector<bool> used(free_pos.size(), false);
    for (int r = 0; r < nslot; ++r) {
        for (size_t i = 0; i < free_pos.size(); ++i) {
            if (!used[i] && tile_slot_bit(free_pos[i], elem_bytes, access) == r) {
                head.push_back(free_pos[i]);
                used[i] = true;
                break;
            }
        }
    }
    for (size_t i = 0; i < free_pos.size(); ++i)
        if (!used[i]) rest.push_back(free_pos[i]);
    free_pos = head;
    free_pos.insert(free_pos.end(), rest.begin(), rest.end());
}

// Order in which free tile positions pad a round's register set: positions
// that select no slot bit first, then ascending, position 0 last (for 8-byte
// elements it is the only position on slot bit 0).
std::vector<int> register_pad_order(int T, int elem_bytes) {
    std::vector<int> o;
    for (int p = 1; p < T; ++p)
        if (tile_slot_bit(p, elem_bytes, elem_bytes) < 0) o.push_back(p);
    for (int p = 1; p < T; ++p)
        if (tile_slot_bit(p, elem_bytes, elem_bytes) >= 0) o.push_back(p);
    o.push_back(0);
    return o;
}

// A gop for scheduling: the qubits it acts on diagonally, as X and otherwise
// (gop_actions), and its non-diagonal targets.
struct SchedOp {
    uint64_t z = 0, x = 0, g = 0, targets = 0;
    bool tile = true;   // can join a tile pass
    bool round = true;  // can join a register round
    bool probe = false;
};

SchedOp sched_op(const GOp& g) {
    SchedOp s;
    std::vector<std::pair<int, uint8_t>> acts;
    std::vector<int> targ;
    gop_actions(g, &acts);
    for (auto& a : acts) (a.second == A_Z ? s.z : (a.second == A_X ? s.x : s.g)) |= 1ULL << a.first;
    gop_targets(g, &targ);
    for (int t : targ) s.targets |= 1ULL << t;
    s.tile = g.kind != K_DENSEK;
    s.round = g.kind != K_DENSE2;
    s.probe = g.kind == K_PROBE;
    return s;
}

// Operations left out so far, as the actions they block (act_conflict).
struct Blocked {
    uint64_t z = 0, x = 0, g = 0;
    bool conflicts(const SchedOp& o) const { return ((o.z & (x | g)) | (o.x & (z | g)) | (o.g & (z | x | g))) != 0; }
    void add(const SchedOp& o) {
        z |= o.z;
        x |= o.x;
        g |= o.g;
    }
};

// How many of the first `window` operations of `todo` can run together, in
// order, when the non-diagonal targets are limited to `allowed`.
int count_joining(const std::vector<SchedOp>& ops, const std::vector<int>& todo, uint64_t allowed, bool round,
                  size_t window, int cap) {
    Blocked b;
    int joined = 0;
    const size_t m = std::min(window, todo.size());
    for (size_t i = 0; i < m && joined < cap; ++i) {
        const SchedOp& o = ops[static_cast<size_t>(todo[i])];
        if ((round ? o.round : o.tile) && !(o.targets & ~allowed) && !b.conflicts(o)) ++joined;
        else b.add(o);
    }
    return joined;
}

// Local search for the qubits that let the most operations join: from
// `start`, the best exchange of one qubit for another of `from` until none
// improves the count.
uint64_t best_set(const std::vector<SchedOp>& ops, const std::vector<int>& todo, uint64_t fixed, uint64_t start,
                  uint64_t from, bool round, size_t window, int cap) {
    uint64_t set = start;
    int best = count_joining(ops, todo, fixed | set, round, window, cap);
    for (;;) {
        uint64_t next = set;
        for (uint64_t out = set; out && best < cap; out &= out - 1)
            for (uint64_t in = from & ~set; in; in &= in - 1) {
                const uint64_t c = (set & ~(out & (~out + 1))) | (in & (~in + 1));
                const int v = count_joining(ops, todo, fixed | c, round, window, cap);
                if (v > best) {
                    best = v;
                    next = c;
                }
            }
        if (next == set) return set;
        set = next;
    }
}

// The sets chosen for a circuit's passes and rounds, in order.  They depend on
// the circuit's structure alone, and finding them costs milliseconds (30 qubits,
// 1800 gates: 15 ms, then 1.6), so re-planning a structure at other angles looks them
// up: the last PLAN_CHOICES structures of the process, up to
// PLAN_CHOICE_BYTES of keys and sets, keyed by every field the search reads.
struct Choices {
    std::vector<uint64_t> sets;
};
constexpr size_t PLAN_CHOICES = 32;
constexpr size_t PLAN_CHOICE_BYTES = 16 << 20;

std::mutex g_choices_mu;
std::list<std::pair<std::string, Choices>> g_choices;  // most recent first
size_t g_choice_bytes = 0;

size_t choice_bytes(const std::pair<std::string, Choices>& c) {
    return c.first.capacity() + c.second.sets.capacity() * sizeof(uint64_t);
}

std::string choices_key(int n, int eb, int T, int R, int cap, const std::vector<SchedOp>& ops) {
    std::string k;
    k.reserve(ops.size() * 36 + 16);
    auto put = [&](const auto& v) { k.append(reinterpret_cast<const char*>(&v), sizeof v); };
    put(n);
    put(eb);  // the registers' padding (register_pad_order)
    put(T);
    put(R);
    put(cap);
    for (const SchedOp& o : ops) {
        put(o.z);
        put(o.x);
        put(o.g);
        put(o.targets);
        k.push_back(static_cast<char>(o.tile | o.round << 1 | o.probe << 2));
    }
    return k;
}

bool find_choices(const std::string& key, Choices* c) {
    std::lock_guard<std::mutex> lk(g_choices_mu);
    for (auto it = g_choices.begin(); it != g_choices.end(); ++it)
        if (it->first == key) {
            g_choices.splice(g_choices.begin(), g_choices, it);
            *c = it->second;
            return true;
        }
    return false;
}

void keep_choices(std::string key, Choices c) {
    std::lock_guard<std::mutex> lk(g_choices_mu);
    for (const auto& kept : g_choices)
        if (kept.first == key) return;  // another thread planned it meanwhile
    g_choices.emplace_front(std::move(key), std::move(c));
    g_choice_bytes += choice_bytes(g_choices.front());
    while (!g_choices.empty() && (g_choices.size() > PLAN_CHOICES || g_choice_bytes > PLAN_CHOICE_BYTES)) {
        g_choice_bytes -= choice_bytes(g_choices.back());
        g_choices.pop_back();
    }
}

// Operations of one tile pass at most.  Fewer and larger passes are faster up
// to where their unrolled code leaves the instruction cache, and that shows only
// where a pass streams far more than the L2.  Complex64 (13, 5), depth 20 and 40
// (us): 14 qubits 85 and 164 at 45 operations, 62 and 110 at 130 or without a
// limit; 20 qubits 137 and 251, 118 and 206; 25 qubits 2048 and 3844, 1798 and
// 3489; 27 qubits 7988 and 15595 at 45, 7510 and 14193 at 62, 8051 and 14462 at
// 130.  128 rather than no limit bounds the compilation, which grows faster than
// the pass (13 qubits: 760 operations 4 s, 3800 in one pass 48 s).
// Reverse sweeps do not depend on it (11 to 22 qubits: 2%), batched ones take
// any number (23.3 ms at 42, 21.3 at 62, 19.1 without).  Above 26 qubits and for
// sweeps the limits are lower than that asks for: tests/test_jit_host.py bounds
// the code size over at least 40 passes of two benchmark circuits.
int pass_op_cap(int n, int R, bool two_states, bool bound) {
    if (bound) return INT_MAX;
    if (two_states) return R <= 3 ? 84 : 62;
    if (R < 5) return INT_MAX;
    return n > 26 ? 45 : 128;
}

}  // namespace

bool build_plan(int n, int precision, const std::vector<GOp>& gops, int T, int R, HostPlan* plan,
                std::string* err) {
    *plan = HostPlan();
    plan->n = n;
    plan->precision = precision;
    if (n < 1 || n > QFVM_MAX_QUBITS) {
        *err = "qubit count " + std::to_string(n) + " outside 1.." + std::to_string(QFVM_MAX_QUBITS);
        return false;
    }
    int dT, dR;
    default_shape(n, precision, &dT, &dR);
    if (T <= 0) T = dT;
    if (R <= 0) R = dR;
    if (T < 6 || T > MAX_TILE || R < 2 || R > 6 || R >= T) {
        *err = "invalid tile shape";
        return false;
    }
    const double Sb = amp_bytes(precision);
    const double N = std::ldexp(1.0, n);
    PlanStats& st = plan->stats;
    st.gates = static_cast<int64_t>(gops.size());
    for (const auto& g : gops) st.gate_bytes += gop_bytes(g, n, precision);

    // Small states: one whole-state pass with every gate in order.
    if (n < T) {
        if (n > small_max_qubits(precision)) {
            *err = "state too large for the whole-state kernel";
            return false;
        }
        // runs of gates become whole-state passes; a dense gate on more than
        // MAXK targets (beyond the whole-state kernel's registers) runs as its
        // own global pass between them
        size_t gi = 0;
        while (gi < gops.size()) {
            PassDesc pd;
            std::memset(&pd, 0, sizeof(pd));
            pd.T = n;
            pd.op_begin = static_cast<int32_t>(plan->ops.size());
            pd.probe_base = static_cast<int32_t>(plan->probe_slot.size());
            if (gops[gi].kind == K_DENSEK && gops[gi].k > MAXK) {
                pd.type = PASS_GLOBALOP;
                plan->ops.push_back(global_kop(plan, gops[gi]));
                ++gi;
            } else {
                pd.type = PASS_SMALL;
                while (gi < gops.size() && !(gops[gi].kind == K_DENSEK && gops[gi].k > MAXK))
                    plan->ops.push_back(global_kop(plan, gops[gi++]));
            }
            pd.op_count = static_cast<int32_t>(plan->ops.size()) - pd.op_begin;
            pd.nprobe = static_cast<int32_t>(plan->probe_slot.size()) - pd.probe_base;
            plan->passes.push_back(pd);
            st.passes += 1;
            st.pass_bytes += 2.0 * Sb * N;
        }
        st.rounds = 0;
        plan->T = n;
        plan->R = 0;
        plan->L = n;
        while (plan->coef.size() % 4) plan->coef.push_back(0.0);  // 4-wide reads of the last block
        return true;
    }

    const int L = std::min(5, T - 1);
    const int H = T - L;
    plan->T = T;
    plan->R = R;
    plan->L = L;
    const int eb = amp_bytes(precision);  // element bytes of the shared-memory tile
    const std::vector<int> pad_order = register_pad_order(T, eb);

    std::vector<int> pending(gops.size());
    for (size_t i = 0; i < gops.size(); ++i) pending[i] = static_cast<int>(i);
    std::vector<SchedOp> sops;
    sops.reserve(gops.size());
    bool two_states = false, bound = false;
    for (const GOp& g : gops) {
        sops.push_back(sched_op(g));
        two_states |= g.kind == K_PROBE;
        bound |= g.bkind != 0 && g.slot >= 0 && g.kind != K_PROBE;
    }
    const int cap = pass_op_cap(n, R, two_states, bound);
    const uint64_t low = (1ULL << L) - 1, every = n >= 64 ? ~0ULL : (1ULL << n) - 1;
    std::string key = choices_key(n, eb, T, R, cap, sops);
    Choices choices;
    const bool known = find_choices(key, &choices);
    size_t next_choice = 0;
    // the k lowest bits of m
    auto lowest = [](uint64_t m, int k) {
        uint64_t r = 0;
        for (; k > 0 && m; --k, m &= m - 1) r |= m & (~m + 1);
        return r;
    };
    constexpr size_t WINDOW = 384;  // pending operations the search looks ahead

    while (!pending.empty()) {
        // ---- choose the tile's high qubits and the gates of this pass ----
        uint64_t high = 0;  // global qubits >= L in the tile
        if (known) {
            high = choices.sets[next_choice++];
        } else {
            // in order of the gates' first need, then by local search
            Blocked b;
            for (int gi : pending) {
                const SchedOp& o = sops[static_cast<size_t>(gi)];
                const uint64_t need = high | (o.targets & ~low);
                if (o.tile && !b.conflicts(o) && __builtin_popcountll(need) <= H) high = need;
                else b.add(o);
            }
            high |= lowest(every & ~low & ~high, H - __builtin_popcountll(high));
            high = best_set(sops, pending, low, high, every & ~low, false, WINDOW, cap);
            choices.sets.push_back(high);
        }
        std::vector<int> sched, rest;
        {
            Blocked b;
            int probes = 0;
            for (int gi : pending) {
                const SchedOp& o = sops[static_cast<size_t>(gi)];
                const bool ok = o.tile && !(o.targets & ~(low | high)) && !b.conflicts(o) &&
                                static_cast<int>(sched.size()) < cap && (!o.probe || probes < MAX_PASS_PROBES);
                if (ok) {
                    sched.push_back(gi);
                    probes += o.probe;
                } else {
                    b.add(o);
                    rest.push_back(gi);
                }
            }
        }
        if (sched.empty()) {
            // The first pending gate cannot join a tile pass (a dense gate on
            // more than two targets): apply it on its own.
            const int gi = pending.front();
            PassDesc pd;
            std::memset(&pd, 0, sizeof(pd));
            pd.type = PASS_GLOBALOP;
            pd.op_begin = static_cast<int32_t>(plan->ops.size());
            pd.op_count = 1;
            plan->ops.push_back(global_kop(plan, gops[gi]));
            plan->passes.push_back(pd);
            st.passes += 1;
            st.pass_bytes += 2.0 * Sb * N;
            pending.erase(pending.begin());
            continue;
        }
        PassDesc pd;
        std::memset(&pd, 0, sizeof(pd));
        pd.type = PASS_TILE;
        pd.T = T;
        pd.L = L;
        pd.H = H;
        int local_of[64];
        for (int q = 0; q < 64; ++q) local_of[q] = -1;
        for (int k = 0; k < L; ++k) {
            pd.tq[k] = static_cast<uint8_t>(k);
            local_of[k] = k;
        }
        {
            int k = L;
            for (uint64_t m = high; m; m &= m - 1, ++k) {
                const int q = __builtin_ctzll(m);
                pd.tq[k] = static_cast<uint8_t>(q);
                local_of[q] = k;
            }
        }
        pd.step_begin = static_cast<int32_t>(plan->steps.size());
        pd.probe_base = static_cast<int32_t>(plan->probe_slot.size());

        // ---- split the pass's gates into register rounds ----
        // Two-target dense gates run as shared-memory steps of the tile (in
        // order); everything else runs in register rounds.
        std::vector<int> todo = sched;
        while (!todo.empty()) {
            if (gops[todo.front()].kind == K_DENSE2) {
                const GOp& g = gops[todo.front()];
                StepDesc sd;
                std::memset(&sd, 0, sizeof(sd));
                sd.type = STEP_SMEM;
                sd.op_begin = static_cast<int32_t>(plan->ops.size());
                sd.op_count = 1;
                KOp ko;
                std::memset(&ko, 0, sizeof(ko));
                ko.kind = g.kind;
                ko.t0 = static_cast<uint8_t>(local_of[g.t0]);
                ko.t1 = static_cast<uint8_t>(local_of[g.t1]);
                for (int q = 0; q < n; ++q) {
                    const uint64_t b = 1ULL << q;
                    if (g.cmask & b) {
                        if (local_of[q] >= 0) ko.creg |= 1u << local_of[q];
                        else ko.cthr |= b;
                    }
                }
                ko.coef = push_coef(plan, g);
                plan->ops.push_back(ko);
                plan->steps.push_back(sd);
                st.rounds += 1;
                todo.erase(todo.begin());
                continue;
            }
            uint64_t rset = 0;  // the register bits' global qubits
            if (known) {
                rset = choices.sets[next_choice++];
            } else {
                Blocked b;
                for (int gi : todo) {
                    const SchedOp& o = sops[static_cast<size_t>(gi)];
                    const uint64_t need = rset | o.targets;
                    if (o.round && !b.conflicts(o) && __builtin_popcountll(need) <= R) rset = need;
                    else b.add(o);
                }
                // pad the register set (register_pad_order)
                for (size_t x = 0; x < pad_order.size() && __builtin_popcountll(rset) < R; ++x)
                    rset |= 1ULL << pd.tq[pad_order[x]];
                rset = best_set(sops, todo, 0, rset, low | high, true, todo.size(), static_cast<int>(todo.size()));
                choices.sets.push_back(rset);
            }
            std::vector<int> regs;  // tile-local positions
            for (uint64_t m = rset; m; m &= m - 1) regs.push_back(local_of[__builtin_ctzll(m)]);
            std::vector<int> round_ops, left;
            {
                Blocked b;
                for (int gi : todo) {
                    const SchedOp& o = sops[static_cast<size_t>(gi)];
                    if (o.round && !(o.targets & ~rset) && !b.conflicts(o)) {
                        round_ops.push_back(gi);
                    } else {
                        b.add(o);
                        left.push_back(gi);
                    }
                }
            }
            StepDesc sd;
            std::memset(&sd, 0, sizeof(sd));
            sd.type = STEP_ROUND;
            for (int k = 0; k < R; ++k) sd.rpos[k] = static_cast<uint8_t>(regs[k]);
            std::vector<int> freep;
            for (int p = 0; p < T; ++p)
                if (std::find(regs.begin(), regs.end(), p) == regs.end()) freep.push_back(p);
            // 8-byte elements with position 0 in the registers: the specialised
            // passes access the register pairs (j, j | bit of position 0) 16 bytes at a time
            const bool pairs = eb == 8 && std::find(regs.begin(), regs.end(), 0) != regs.end();
            order_thread_bits(freep, eb, pairs ? 16 : eb);
            const uint32_t u = 16u / static_cast<uint32_t>(eb);
            for (size_t k = 0; k < freep.size(); ++k) {
                sd.tpos[k] = static_cast<uint8_t>(freep[k]);
                sd.tglob[k] = pd.tq[freep[k]];
                sd.tsw[k] = static_cast<uint16_t>(tile_weight(freep[k], u));
            }
            for (int k = 0; k < R; ++k) sd.rsw[k] = static_cast<uint16_t>(tile_weight(regs[k], u));
            int reg_of_local[MAX_TILE];
            for (int p = 0; p < MAX_TILE; ++p) reg_of_local[p] = -1;
            for (int k = 0; k < R; ++k) reg_of_local[regs[k]] = k;
            sd.op_begin = static_cast<int32_t>(plan->ops.size());
            for (int gi : round_ops) {
                const GOp& g = gops[gi];
                KOp ko;
                std::memset(&ko, 0, sizeof(ko));
                ko.kind = g.kind;
                ko.flags = g.flags;
                ko.special = g.special;
                if (g.t0 >= 0) ko.t0 = static_cast<uint8_t>(reg_of_local[local_of[g.t0]]);
                if (g.t1 >= 0) ko.t1 = static_cast<uint8_t>(reg_of_local[local_of[g.t1]]);
                for (int q = 0; q < n; ++q) {
                    const uint64_t b = 1ULL << q;
                    const int lp = local_of[q];
                    const int rb = (lp >= 0) ? reg_of_local[lp] : -1;
                    if (g.cmask & b) {
                        if (rb >= 0) ko.creg |= 1u << rb;
                        else ko.cthr |= b;
                    }
                    if (g.pmask & b) {
                        if (rb >= 0) ko.preg |= 1u << rb;
                        else ko.pthr |= b;
                    }
                }
                if (ko.cthr) ko.flags |= F_TCTRL;
                if (ko.pthr) ko.flags |= F_TPAR;
                if (g.kind == K_PROBE) {
                    for (int q = 0; q < n; ++q)
                        if (g.xmask & (1ULL << q)) ko.xreg |= 1u << reg_of_local[local_of[q]];
                    ko.probe = static_cast<uint16_t>(plan->probe_slot.size() - pd.probe_base);
                    plan->probe_slot.push_back(g.slot);
                }
                if (g.kind == K_DIAG && ko.creg == 0) {
                    if (ko.preg == 0) {
                        ko.flags |= F_UNIFORM;  // one factor per thread, folded into the round phase
                    } else if (__builtin_popcount(ko.preg) == 1) {
                        ko.flags |= F_ONEBIT;
                        ko.t0 = static_cast<uint8_t>(__builtin_ctz(ko.preg));
                    }
                }
                ko.coef = push_coef(plan, g);
                plan->ops.push_back(ko);
            }
            sd.op_count = static_cast<int32_t>(round_ops.size());
            plan->steps.push_back(sd);
            st.rounds += 1;
            todo = left;
        }
        pd.step_count = static_cast<int32_t>(plan->steps.size()) - pd.step_begin;
        pd.nprobe = static_cast<int32_t>(plan->probe_slot.size()) - pd.probe_base;
        plan->passes.push_back(pd);
        st.passes += 1;
        st.pass_bytes += 2.0 * Sb * N;
        pending = rest;
    }
    if (!known) keep_choices(std::move(key), std::move(choices));
    while (plan->coef.size() % 4) plan->coef.push_back(0.0);  // 4-wide reads of the last block
    return true;
}

GOp gop_dagger(const GOp& g) {
    GOp d = g;
    d.bsign = static_cast<int8_t>(-g.bsign);
    auto conj_transpose = [&](int dim) {
        std::vector<double> c(g.coef.size());
        for (int r = 0; r < dim; ++r)
            for (int k = 0; k < dim; ++k) {
                c[2 * (r * dim + k)] = g.coef[2 * (k * dim + r)];
                c[2 * (r * dim + k) + 1] = -g.coef[2 * (k * dim + r) + 1];
            }
        d.coef = c;
    };
    switch (g.kind) {
        case K_REAL: d.coef = {g.coef[0], g.coef[2], g.coef[1], g.coef[3]}; break;  // real unitary: transpose
        case K_RX: d.coef = {g.coef[0], -g.coef[1]}; break;
        case K_DENSE: conj_transpose(2); break;
        case K_DENSE2: conj_transpose(4); break;
        case K_DENSEK: conj_transpose(1 << g.k); break;
        case K_DIAG:
            d.coef = {g.coef[0], -g.coef[1], g.coef[2], -g.coef[3]};
            if (g.flags & F_D1_SPEC) {
                if (g.special == SP_I) d.special = SP_NEGI;
                else if (g.special == SP_NEGI) d.special = SP_I;
            }
            break;
        default: break;  // X, Y, SWAP are self-inverse
    }
    return d;
}

bool build_adjoint_sweep(const std::vector<GOp>& gops, std::vector<GOp>* out, std::string* err) {
    out->clear();
    out->reserve(gops.size() * 2);
    for (size_t r = gops.size(); r-- > 0;) {
        const GOp& g = gops[r];
        if (g.slot >= 0) {
            if (!g.has_gen) {
                *err = "op " + std::to_string(g.src) + " carries a parameter slot but has no generator";
                return false;
            }
            GOp pr;
            pr.kind = K_PROBE;
            pr.xmask = g.gx;
            pr.pmask = g.gz;
            pr.cmask = g.gcmask;
            pr.special = static_cast<uint8_t>(g.gny & 3);
            pr.coef = {g.gscale};
            pr.slot = g.slot;
            pr.src = g.src;
            out->push_back(pr);
        }
        out->push_back(gop_dagger(g));
    }
    return true;
}

int bind_coef(int kind, double th, double* c) {
    switch (kind) {
        case QFVM_OP_RX:
            c[0] = std::cos(th / 2);
            c[1] = std::sin(th / 2);
            return 2;
        case QFVM_OP_RY:
            c[0] = std::cos(th / 2);
            c[1] = -std::sin(th / 2);
            c[2] = std::sin(th / 2);
            c[3] = std::cos(th / 2);
            return 4;
        case QFVM_OP_RZ:
        case QFVM_OP_RZZ:
            c[0] = std::cos(-th / 2);
            c[1] = std::sin(-th / 2);
            c[2] = std::cos(th / 2);
            c[3] = std::sin(th / 2);
            return 4;
        case QFVM_OP_P:
        case QFVM_OP_CP:
            c[0] = 1.0;
            c[1] = 0.0;
            c[2] = std::cos(th);
            c[3] = std::sin(th);
            return 4;
        default: return 0;
    }
}

bool unfix_bound(std::vector<GOp>* gops, std::string* err) {
    for (GOp& g : *gops) {
        if (g.slot < 0) continue;
        if (g.bkind == 0) {
            *err = "op " + std::to_string(g.src) +
                   ": only rx/ry/rz/p/cp/rzz gates can carry a per-item parameter in a batched run";
            return false;
        }
        if (g.kind == K_DIAG) {
            g.flags &= static_cast<uint8_t>(~F_D1_SPEC);
            g.special = 0;
            if (g.bkind == QFVM_OP_RZ || g.bkind == QFVM_OP_RZZ) {
                g.flags &= static_cast<uint8_t>(~F_D0_ONE);
                g.special = SP_BOUND_RZ;
            }
        }
    }
    return true;
}

namespace {

bool is_plain_hadamard(const GOp& g) {
    const double h = 1. / std::sqrt(2.);
    return g.kind == K_REAL && g.cmask == 0 && g.slot < 0 && g.bkind == 0 && g.coef.size() == 4 &&
           g.coef[0] == h && g.coef[1] == h && g.coef[2] == h && g.coef[3] == -h;
}

// a gate that touches every amplitude through its coefficients alone, so a
// scalar multiplies into them exactly where it would multiply the state
bool can_absorb_scalar(const GOp& g) {
    if (g.cmask != 0 || g.slot >= 0 || g.bkind != 0) return false;
    if (g.kind == K_REAL || g.kind == K_RX || g.kind == K_DENSE) return !is_plain_hadamard(g);
    if (g.kind == K_DIAG) return (g.flags & (F_D0_ONE | F_D1_SPEC)) == 0;
    return false;
}

void scale_coefs(GOp& g, int halves) {
    // (1/sqrt(2))^halves = 2^(-halves/2), one rounding when halves is odd
    double f = std::ldexp(1.0, -(halves / 2));
    if (halves & 1) f *= 1. / std::sqrt(2.);
    for (double& c : g.coef) c *= f;
}

}  // namespace

bool known_unitary(const qfvm_op* ops, int64_t n_ops, const double* matpool) {
    constexpr double TOL = 1e-9;  // far below complex64's rounding
    for (int64_t i = 0; i < n_ops; ++i) {
        if (ops[i].kind != QFVM_OP_MATRIX) continue;  // the named gates are
        const int64_t dim = ops[i].mat_dim;
        if (dim > (1 << MAXK)) return false;
        const cd* m = reinterpret_cast<const cd*>(matpool) + ops[i].mat_offset;
        for (int64_t a = 0; a < dim; ++a)
            for (int64_t b = a; b < dim; ++b) {  // columns a and b
                cd s(a == b ? -1.0 : 0.0, 0.0);
                for (int64_t r = 0; r < dim; ++r) s += std::conj(m[r * dim + a]) * m[r * dim + b];
                if (!(std::abs(s) <= TOL)) return false;
            }
    }
    return true;
}

namespace {

uint64_t targets_of(const GOp& g) {
    uint64_t m = 0;
    if (g.t0 >= 0) m |= 1ULL << g.t0;
    if (g.t1 >= 0) m |= 1ULL << g.t1;
    if (g.kind == K_DENSEK)
        for (int j = 0; j < g.k; ++j) m |= 1ULL << g.tk[j];
    return m;
}
uint64_t touches(const GOp& g) { return g.cmask | g.pmask | targets_of(g); }

enum MergeClass { M_NONE, M_DIAG, M_RX, M_X };
MergeClass merge_class(const GOp& g) {
    if (g.cmask != 0 || g.slot >= 0 || g.bkind != 0) return M_NONE;
    if (g.kind == K_DIAG && g.pmask != 0 && (g.pmask & (g.pmask - 1)) == 0 && g.coef.size() == 4) return M_DIAG;
    if (g.kind == K_RX && g.coef.size() == 2) return M_RX;
    if (g.kind == K_X) return M_X;
    return M_NONE;
}

// whether a one-qubit gate of class c on qubit bit qb commutes with p (which
// touches qb): diagonals commute with diagonals and with gates that use qb
// only as a control; X-type gates commute with X / RX on the same target
bool commutes(MergeClass c, uint64_t qb, const GOp& p) {
    if (c == M_DIAG) return p.kind == K_DIAG || ((p.cmask & qb) && !(p.pmask & qb) && !(targets_of(p) & qb));
    return (p.kind == K_X || p.kind == K_RX) && p.t0 >= 0 && (1ULL << p.t0) == qb && !(p.cmask & qb);
}

}  // namespace

void fuse_single_qubit(std::vector<GOp>* gops) {
    constexpr int MAX_SCAN = 512;
    std::vector<GOp>& g = *gops;
    std::vector<char> dead(g.size(), 0);
    for (size_t j = 0; j < g.size(); ++j) {
        const MergeClass c = merge_class(g[j]);
        if (c == M_NONE) continue;
        const uint64_t qb = c == M_DIAG ? g[j].pmask : (1ULL << g[j].t0);
        int scanned = 0;
        for (size_t i = j; i-- > 0 && scanned < MAX_SCAN; ++scanned) {
            if (dead[i] || !(touches(g[i]) & qb)) continue;
            GOp& a = g[i];
            if (merge_class(a) == c && (c == M_DIAG ? a.pmask == qb : (1ULL << a.t0) == qb)) {
                if (c == M_DIAG) {
                    const cd d0 = cd(a.coef[0], a.coef[1]) * cd(g[j].coef[0], g[j].coef[1]);
                    const cd d1 = cd(a.coef[2], a.coef[3]) * cd(g[j].coef[2], g[j].coef[3]);
                    a.flags &= static_cast<uint8_t>(~(F_D0_ONE | F_D1_SPEC));
                    a.special = 0;
                    set_diag(a, d0, d1);
                } else if (c == M_RX) {
                    // rx(a) rx(b) = rx(a + b): [[c, -is], [-is, c]]
                    const double c1 = a.coef[0], s1 = a.coef[1], c2 = g[j].coef[0], s2 = g[j].coef[1];
                    a.coef = {c1 * c2 - s1 * s2, s1 * c2 + c1 * s2};
                } else {
                    dead[i] = 1;  // X X = I
                }
                dead[j] = 1;
                break;
            }
            if (!commutes(c, qb, a)) break;
        }
    }
    size_t w = 0;
    for (size_t i = 0; i < g.size(); ++i)
        if (!dead[i]) g[w++] = g[i];
    g.resize(w);
}

void unnormalize_hadamards(std::vector<GOp>* gops) {
    // |amplitudes| stay below 2^64 between absorptions: with the 2^48 of
    // normalize_passes (NORM_ONE_STATE) on top, FP32 holds them
    constexpr int MAX_PENDING = 128;
    std::vector<size_t> pending;
    int last = -1;
    for (size_t i = 0; i < gops->size(); ++i) {
        GOp& g = (*gops)[i];
        if (is_plain_hadamard(g) && static_cast<int>(pending.size()) < MAX_PENDING) {
            pending.push_back(i);
        } else if (can_absorb_scalar(g)) {
            if (!pending.empty()) {
                scale_coefs(g, static_cast<int>(pending.size()));
                for (size_t k : pending) {
                    (*gops)[k].kind = K_HAD;
                    (*gops)[k].coef.clear();
                }
                pending.clear();
            }
            last = static_cast<int>(i);
        }
    }
    if (!pending.empty() && last >= 0) {
        // a global scalar commutes with every gate: an earlier gate takes it
        scale_coefs((*gops)[static_cast<size_t>(last)], static_cast<int>(pending.size()));
        for (size_t k : pending) {
            (*gops)[k].kind = K_HAD;
            (*gops)[k].coef.clear();
        }
    }
}

void simplify_plain(std::vector<GOp>* gops) {
    for (GOp& g : *gops) {
        g.slot = -1;
        g.bkind = 0;
    }
    fuse_single_qubit(gops);
    unnormalize_hadamards(gops);
}

namespace {

// Scalars taken out of a pass's gates (normalize_passes): at most `count` in
// a row before one gate takes their product back, and down to `total`.
// Amplitudes grow by the inverse until the scalar is put back (and shrink by
// as much where the gate that takes it comes first), so the limits keep them
// and the low halves of float pairs inside FP32's exponents (2^-149 to 2^128):
//   one state: 2^48 leaves a factor of 2^80 to an input state far from
//     normalised, and to Hadamards without their 1/sqrt(2);
//   reverse sweep: a probe multiplies two states and its coefficient is
//     divided by the square: 2^72 leaves 2^56 to an observable, a coefficient's
//     low half is 2^-121 then, and average products of 30 qubits shrunk by as
//     much (2^-102) still have the 47 bits of a float pair.
// A gate whose scalar is below NORM_MIN is left as it is.
//
// Passes that differ only in their angles have to share one compiled kernel,
// and a kernel depends on which gates are in unit form.  So every group of a
// pass gives up all its scalars but one, or, where a group's product is beyond
// the limit, every second rotation of the pass its own: two patterns a pass
// (gate by gate up to the limit, a circuit near pi met new patterns at almost
// every step of a training).  At random angles a scalar is about 1/2 in the
// geometric mean: 4e-8 of the gates are below NORM_MIN, 4e-6 (one state) and
// 4e-5 (sweep) of the groups beyond their limit.
struct NormLimits {
    int count;
    double total;
};
constexpr NormLimits NORM_ONE_STATE = {15, 0x1p-48}, NORM_SWEEP = {11, 0x1p-36};
constexpr double NORM_MIN = 0x1p-24;

bool uncontrolled(const KOp& o) { return o.cthr == 0 && o.creg == 0; }

// Numbers of 106 bits as the sum of two doubles (TwoSum, TwoProd with FMA;
// Dekker 1971, Ogita, Rump and Oishi 2005).  (long double would do, but is
// software on Arm: 24 qubits, 960 parameters, 2 ms a call.)
struct Dd {
    double h = 0.0, l = 0.0;
};
Dd two_sum(double a, double b) {
    const double s = a + b, v = s - a;
    return {s, (a - (s - v)) + (b - v)};
}
Dd two_prod(double a, double b) {
    const double p = a * b;
    return {p, std::fma(a, b, -p)};
}
Dd operator+(Dd a, Dd b) {
    const Dd s = two_sum(a.h, b.h);
    return two_sum(s.h, s.l + (a.l + b.l));
}
Dd operator-(Dd a) { return {-a.h, -a.l}; }
Dd operator*(Dd a, Dd b) {
    const Dd p = two_prod(a.h, b.h);
    return two_sum(p.h, p.l + std::fma(a.h, b.l, a.l * b.h));
}
Dd operator/(Dd a, Dd b) {
    const double q = a.h / b.h;
    const Dd r = a + -(b * Dd{q, 0.0});
    return two_sum(q, r.h / b.h);
}

struct Scalar {
    Dd re, im;
    double abs() const { return std::hypot(re.h, im.h); }
    double norm() const { return re.h * re.h + im.h * im.h; }
    bool one() const { return re.h == 1.0 && re.l == 0.0 && im.h == 0.0; }
};
Scalar operator*(const Scalar& a, const Scalar& b) {
    if (a.im.h == 0.0 && b.im.h == 0.0) return {a.re * b.re, {}};
    return {a.re * b.re + -(a.im * b.im), a.re * b.im + a.im * b.re};
}

// 1 / |(1, t)|, the scalar that leaves a rotation with off-diagonal entries t
// and -t (or -it and -it) unitary whatever t was rounded to (one Newton step
// from c); c itself where the gate is not a rotation
Dd rotation_scalar(double c, double s) {
    if (!(std::fabs(c * c + s * s - 1.0) < 0x1p-48)) return {c, 0.0};
    const Dd ct = two_prod(c, s / c);
    const Dd r = Dd{1.0, 0.0} + -(two_prod(c, c) + ct * ct);
    return two_sum(c, 0.5 * c * r.h);
}

// a rotation with equal diagonal entries, or a two-valued phase of register
// bits: the scalar that makes its first diagonal entry 1.  Rounded to double
// one product after the other, they were the largest error of an FP64 plan
// beside the amplitudes' own roundings.
bool scalar_of(const KOp& o, const double* c, Scalar* f) {
    if (!uncontrolled(o)) return false;
    double size = 0.0;
    if (o.kind == K_REAL || o.kind == K_RX) {
        if (o.kind == K_REAL && c[0] != c[3]) return false;
        size = std::fabs(c[0]);
    } else if (o.kind == K_DIAG) {
        if (o.flags & (F_D0_ONE | F_D1_SPEC | F_UNIFORM | F_TPAR)) return false;
        size = std::hypot(c[0], c[1]);
    } else {
        return false;
    }
    if (!(size >= NORM_MIN && size <= 1.0 / NORM_MIN)) return false;
    *f = Scalar{};
    if (o.kind == K_RX) f->re = rotation_scalar(c[0], c[1]);
    else if (o.kind == K_REAL) f->re = c[1] == -c[2] ? rotation_scalar(c[0], c[2]) : Dd{c[0], 0.0};
    else *f = Scalar{{c[0], 0.0}, {c[1], 0.0}};
    return true;
}

// number of (complex) coefficients a scalar multiplies into at no cost: the
// op already applies general complex numbers to every amplitude
int free_scalar_coefs(const KOp& o, bool probes) {
    if (!uncontrolled(o)) return 0;
    if (o.kind == K_DENSE) return 4;
    if (o.kind == K_DENSE2) return 16;
    // a phase of thread bits joins the round's phase, which multiplies every
    // amplitude (at the round's end: too late for probes of the same round)
    if (!probes && o.kind == K_DIAG && (o.flags & F_UNIFORM) && (o.flags & F_TPAR) && !(o.flags & (F_D0_ONE | F_D1_SPEC))) return 2;
    return 0;
}

// A pass's operations in order, with their scalars.
struct ScalarOp {
    KOp* o;
    double* c;
    bool has;
    Scalar f;
    double z2;  // factor on |state|^2 from this operation on
};

Scalar product_of_scalars(const std::vector<ScalarOp>& ops, const std::vector<size_t>& from, size_t keeper) {
    Scalar total{{1.0, 0.0}, {}};
    for (size_t i : from)
        if (i != keeper) total = total * ops[i].f;
    return total;
}

bool in_range(const Scalar& z, double least) { return z.abs() >= least && z.abs() <= 1.0 / least; }

// Takes the scalars of `from` (but the keeper's) out and multiplies the keeper
// by their product.
void move_scalars(std::vector<ScalarOp>& ops, const std::vector<size_t>& from, size_t keeper) {
    const Scalar total = product_of_scalars(ops, from, keeper);
    for (size_t i : from) {
        if (i == keeper) continue;
        KOp& o = *ops[i].o;
        double* c = ops[i].c;
        ops[i].z2 /= ops[i].f.norm();
        if (o.kind == K_REAL) {
            c[1] /= c[0];
            c[2] /= c[0];
            c[0] = c[3] = 1.0;
            o.special = SP_UNIT;
        } else if (o.kind == K_RX) {
            c[1] /= c[0];
            c[0] = 1.0;
            o.special = SP_UNIT;
        } else {
            const Scalar conj{ops[i].f.re, -ops[i].f.im};
            const Scalar d1 = Scalar{{c[2], 0.0}, {c[3], 0.0}} * conj;
            const Dd n = ops[i].f.re * ops[i].f.re + ops[i].f.im * ops[i].f.im;
            c[0] = 1.0;
            c[1] = 0.0;
            c[2] = (d1.re / n).h;
            c[3] = (d1.im / n).h;
            o.flags |= F_D0_ONE;
        }
    }
    if (total.one()) return;
    const KOp& o = *ops[keeper].o;
    double* c = ops[keeper].c;
    if (o.kind == K_REAL || o.kind == K_RX) {
        for (int i = 0; i < (o.kind == K_REAL ? 4 : 2); ++i) c[i] = (Dd{c[i], 0.0} * total.re).h;
    } else {
        for (int i = 0; i < (o.kind == K_DIAG ? 2 : free_scalar_coefs(o, false)); ++i) {
            const Scalar v = Scalar{{c[2 * i], 0.0}, {c[2 * i + 1], 0.0}} * total;
            c[2 * i] = v.re.h;
            c[2 * i + 1] = v.im.h;
        }
    }
    ops[keeper].z2 *= total.norm();
}

}  // namespace

void normalize_passes(HostPlan* plan) {
    if (!plan->binds.empty()) return;
    for (const PassDesc& pd : plan->passes) {
        if (pd.type != PASS_TILE) continue;
        std::vector<ScalarOp> ops;
        for (int si = pd.step_begin; si < pd.step_begin + pd.step_count; ++si)
            for (int oi = 0; oi < plan->steps[si].op_count; ++oi) {
                KOp* o = &plan->ops[plan->steps[si].op_begin + oi];
                ScalarOp s{o, plan->coef.data() + o->coef, false, {}, 1.0};
                s.has = scalar_of(*o, s.c, &s.f);
                ops.push_back(s);
            }
        const NormLimits lim = pd.nprobe > 0 ? NORM_SWEEP : NORM_ONE_STATE;
        // the groups, and the op of each that takes the product of the scalars
        // back: one that does so at no cost, else a phase that stays in its
        // full form, else (the product is then real) a rotation
        struct Group {
            std::vector<size_t> diags, rots;
            size_t keeper;
        };
        std::vector<Group> groups;
        bool within = true;
        for (size_t i0 = 0, i1 = 0; i0 < ops.size(); i0 = i1) {
            Group g{{}, {}, ops.size()};
            for (i1 = i0; i1 < ops.size() && static_cast<int>(g.diags.size() + g.rots.size()) <= lim.count; ++i1) {
                if (free_scalar_coefs(*ops[i1].o, pd.nprobe > 0)) g.keeper = i1;
                if (ops[i1].has) (ops[i1].o->kind == K_DIAG ? g.diags : g.rots).push_back(i1);
            }
            if (g.diags.empty() && g.rots.empty()) continue;
            if (g.keeper == ops.size()) g.keeper = !g.diags.empty() ? g.diags.back() : g.rots.back();
            within &= in_range(product_of_scalars(ops, g.rots, g.keeper) * product_of_scalars(ops, g.diags, g.keeper),
                               lim.total);
            groups.push_back(std::move(g));
        }
        for (const Group& g : groups) {
            if (within) {
                std::vector<size_t> all = g.diags;
                all.insert(all.end(), g.rots.begin(), g.rots.end());
                move_scalars(ops, all, g.keeper);
                continue;
            }
            // a phase's scalar is 1 in magnitude where the gate is unitary, a
            // rotation's NORM_MIN at least
            if (!g.diags.empty() && in_range(product_of_scalars(ops, g.diags, g.diags.back()), lim.total / NORM_MIN))
                move_scalars(ops, g.diags, g.diags.back());
            for (size_t k = 0; k + 1 < g.rots.size(); k += 2) move_scalars(ops, {g.rots[k]}, g.rots[k + 1]);
        }
        // reverse sweeps: both states carry the scalars taken out so far, so a
        // probe's sum carries their squared magnitude
        double z = 1.0;
        for (size_t i = 0; i < ops.size() && pd.nprobe > 0; ++i) {
            if (ops[i].o->kind == K_PROBE) *ops[i].c /= z;
            z *= ops[i].z2;
        }
    }
}

std::vector<float> pool_f32(const HostPlan& hp) {
    std::vector<float> out(hp.coef.begin(), hp.coef.end());
    if (!hp.binds.empty()) return out;
    double carry = 1.0;  // exact norm over held norm of the ops so far
    // op's coefficients off .. off + n: scaled by the carry when the op applies
    // them all to every amplitude; either way the rounding's loss is carried on
    auto take = [&](uint32_t off, int n, bool absorbs) {
        const double f = absorbs ? carry : 1.0;
        double exact = 0.0, held = 0.0;
        for (int i = 0; i < n; ++i) {
            const double c = hp.coef[off + i] * f;
            out[off + i] = static_cast<float>(c);
            exact += c * c;
            held += static_cast<double>(out[off + i]) * out[off + i];
        }
        if (held <= 0.0) return;
        carry = (absorbs ? 1.0 : carry) * std::sqrt(exact / held);
    };
    auto visit = [&](const KOp& o) {
        if (o.creg != 0 || (o.kind != K_DIAGR && o.cthr != 0)) return;  // a DIAGR's masks hold its entry codes
        switch (o.kind) {
            case K_REAL: take(o.coef, 4, o.special != SP_UNIT); break;
            case K_RX: take(o.coef, 2, o.special != SP_UNIT); break;
            case K_DENSE: take(o.coef, 8, true); break;
            case K_DENSE2: take(o.coef, 32, true); break;
            case K_DIAG:
                if (!(o.flags & F_D1_SPEC)) take(o.coef, 4, !(o.flags & F_D0_ONE));
                break;
            case K_DIAGR: take(o.coef, 2 << o.k, false); break;
            default: break;
        }
    };
    for (const PassDesc& pd : hp.passes) {
        for (int oi = 0; oi < pd.op_count; ++oi) visit(hp.ops[pd.op_begin + oi]);  // whole-state passes, global ops
        for (int si = pd.step_begin; si < pd.step_begin + pd.step_count; ++si)
            for (int oi = 0; oi < hp.steps[si].op_count; ++oi) visit(hp.ops[hp.steps[si].op_begin + oi]);
    }
    return out;
}

namespace {

// bits of the register index an op of a round acts on non-diagonally
uint32_t nondiag_reg_bits(const KOp& o) {
    switch (o.kind) {
        case K_X: case K_Y: case K_REAL: case K_RX: case K_DENSE: case K_HAD:
            return 1u << o.t0;
        case K_SWAP:
            return (1u << o.t0) | (1u << o.t1);
        case K_DIAG: case K_DIAGR:
            return 0;
        default:
            return ~0u;  // anything else: flush
    }
}

bool mergeable_diag(const KOp& o) {
    return o.kind == K_DIAG && !(o.flags & (F_TCTRL | F_TPAR | F_UNIFORM));
}

int entry_code(cd z) {
    if (z == cd(1.0, 0.0)) return DIAGR_ONE;
    if (z == cd(-1.0, 0.0)) return DIAGR_NEG1;
    if (z == cd(0.0, 1.0)) return DIAGR_I;
    if (z == cd(0.0, -1.0)) return DIAGR_NEGI;
    return DIAGR_GENERAL;
}

}  // namespace

void merge_round_diagonals(HostPlan* plan) {
    // rounds of five register qubits are left alone: their 32-entry tables,
    // and the flips they resolve, measured slower at the complex64 register
    // budget (spills)
    if (plan->R < 1 || plan->R > 4 || !plan->binds.empty() || !plan->probe_slot.empty()) return;
    const int R = plan->R;
    const int NA = 1 << R;
    std::vector<KOp> out;
    out.reserve(plan->ops.size());
    // whole-state passes keep their ops (re-indexed); rounds are rewritten
    std::vector<int32_t> step_begin(plan->steps.size()), step_count(plan->steps.size());
    std::vector<int32_t> pass_begin(plan->passes.size());
    std::vector<bool> step_done(plan->steps.size(), false);
    for (size_t pi = 0; pi < plan->passes.size(); ++pi) {
        PassDesc& pd = plan->passes[pi];
        if (pd.type != PASS_TILE) {
            pass_begin[pi] = static_cast<int32_t>(out.size());
            out.insert(out.end(), plan->ops.begin() + pd.op_begin, plan->ops.begin() + pd.op_begin + pd.op_count);
            continue;
        }
        for (int si = pd.step_begin; si < pd.step_begin + pd.step_count; ++si) {
            const StepDesc& sd = plan->steps[si];
            step_begin[si] = static_cast<int32_t>(out.size());
            step_done[si] = true;
            if (sd.type != STEP_ROUND) {
                out.insert(out.end(), plan->ops.begin() + sd.op_begin, plan->ops.begin() + sd.op_begin + sd.op_count);
                step_count[si] = static_cast<int32_t>(out.size()) - step_begin[si];
                continue;
            }
            std::vector<cd> table(NA, cd(1.0, 0.0));
            std::vector<KOp> merged;
            uint32_t support = 0;
            auto flush = [&]() {
                if (merged.empty()) return;
                if (merged.size() == 1) {
                    out.push_back(merged[0]);
                } else {
                    while (plan->coef.size() % 4) plan->coef.push_back(0.0);
                    KOp k;
                    std::memset(&k, 0, sizeof(k));
                    k.kind = K_DIAGR;
                    k.k = static_cast<uint8_t>(R);
                    k.xreg = support;
                    k.coef = static_cast<uint32_t>(plan->coef.size());
                    for (int j = 0; j < NA; ++j) {
                        plan->coef.push_back(table[j].real());
                        plan->coef.push_back(table[j].imag());
                        const uint64_t c = static_cast<uint64_t>(entry_code(table[j]));
                        if (j < DIAGR_LOW) k.cthr |= c << (3 * j);
                        else k.pthr |= c << (3 * (j - DIAGR_LOW));
                    }
                    out.push_back(k);
                }
                merged.clear();
                std::fill(table.begin(), table.end(), cd(1.0, 0.0));
                support = 0;
            };
            for (int oi = sd.op_begin; oi < sd.op_begin + sd.op_count; ++oi) {
                const KOp& o = plan->ops[oi];
                if (mergeable_diag(o)) {
                    const double* c = plan->coef.data() + o.coef;
                    const cd d0(c[0], c[1]), d1(c[2], c[3]);
                    for (int j = 0; j < NA; ++j) {
                        if ((static_cast<uint32_t>(j) & o.creg) != o.creg) continue;
                        table[j] *= (__builtin_popcount(static_cast<uint32_t>(j) & o.preg) & 1) ? d1 : d0;
                    }
                    support |= o.creg | o.preg;
                    merged.push_back(o);
                    continue;
                }
                if (nondiag_reg_bits(o) & support) flush();
                out.push_back(o);
            }
            flush();
            step_count[si] = static_cast<int32_t>(out.size()) - step_begin[si];
        }
    }
    for (size_t si = 0; si < plan->steps.size(); ++si) {
        if (!step_done[si]) continue;
        plan->steps[si].op_begin = step_begin[si];
        plan->steps[si].op_count = step_count[si];
    }
    for (size_t pi = 0; pi < plan->passes.size(); ++pi)
        if (plan->passes[pi].type != PASS_TILE) plan->passes[pi].op_begin = pass_begin[pi];
    plan->ops.swap(out);
    while (plan->coef.size() % 4) plan->coef.push_back(0.0);
}

}  // namespace qsv
