// Host side of the resident-history lag kernel (lag_hist.cuh): its table and CTA shape.
#pragma once

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "lag_hist.cuh"
#include "lag_host.hpp"

namespace ddm {

// What a launch pairs: register frame j of sub-batch b lives in ring slot reg[b * nreg + j]
// (-1: none); entry i pairs it with window position ent_w[i] + b * nreg + j, whose ring slot is
// pos[...] (-1: none), into accumulator row ent_acc[i]. Window starts ascend strictly.
struct HistInput {
    int nreg = 0, nsub = 1;
    std::vector<int> reg, ent_acc, ent_w, pos;
};

// A table, or why there is none (text). rows is the number of resident rows.
struct HistTable {
    std::vector<int> ints;
    int rows = 0, steps = 0;
    size_t smem = 0;
    long long frames = 0;  // ring frames the launch reads (each once)
};

inline int hist_pick_j(int nreg) {
    for (int J : kHistJs)
        if (J >= nreg) return J;
    return 0;
}

// One unit of work of a thread group: a fused run (kLagFuse entries) or one entry.
struct HistUnit {
    int kind, row, acc, mask;
    double cost() const {  // relative issue slots and shared-memory loads, measured
        return kind == kHistRun ? 3.4 : kind == kHistFull ? 1.0 : 1.5;
    }
};

// Builds the table for blocks of EB elements, CW consumer warps and `buffers` row buffers, with
// register-frame buffers (and stages) or without.
//
// Which entries form fused runs follows build_lag_table's rule exactly (kLagFuse entries in a
// row whose windows are complete and start one position apart, found in order, only for an
// instantiated register-frame count), because a run's sums are formed in another order than a
// single window's: both kernels then give the same bits. Entries without any pair in a
// sub-batch are left out (their accumulators keep their value).
inline std::string build_hist_table(const HistInput &in, int EB, int CW, int buffers, bool x_buffers, HistTable *out) {
    const int nreg = in.nreg, nsub = in.nsub, ntau = static_cast<int>(in.ent_acc.size());
    const int J = hist_pick_j(nreg);
    if (nreg < 1 || J == 0 || nsub < 1 || nsub > kHistMaxSub) return "register frame count out of range";
    if (static_cast<int>(in.reg.size()) < nreg * nsub) return "register frames missing";
    const int npos = static_cast<int>(in.pos.size());
    // pairs that exist
    std::vector<int> mask(static_cast<size_t>(nsub) * ntau, 0);
    std::vector<char> needed(npos, 0);
    const int all = nreg == 32 ? -1 : (1 << nreg) - 1;
    for (int i = 0; i < ntau; i++) {
        if (i > 0 && in.ent_w[i] <= in.ent_w[i - 1]) return "lag windows out of order";
        if (in.ent_w[i] < 0 || in.ent_w[i] + nsub * nreg > npos) return "lag window outside the position table";
    }
    for (int b = 0; b < nsub; b++)
        for (int i = 0; i < ntau; i++) {
            const int w = in.ent_w[i] + b * nreg;
            unsigned m = 0;
            for (int j = 0; j < nreg; j++)
                if (in.reg[b * nreg + j] >= 0 && in.pos[w + j] >= 0) m |= 1u << j;
            mask[static_cast<size_t>(b) * ntau + i] = static_cast<int>(m);
            if (m)
                for (int j = 0; j < nreg; j++) needed[w + j] = 1;
        }
    // the register frames of later sub-batches (without buffers of their own: of all) are read from
    // the resident rows
    const bool in_rows = nsub > 1 || !x_buffers;
    int reg_pos = -1;
    for (int p = 0; p + nsub * nreg <= npos && reg_pos < 0; p++) {
        bool same = true;
        for (int j = 0; j < nsub * nreg && same; j++) same = in.pos[p + j] == in.reg[j];
        if (same) reg_pos = p;
    }
    if (in_rows && reg_pos < 0) return "register frames are not among the positions";
    if (in_rows)
        for (int j = 0; j < nsub * nreg; j++) needed[reg_pos + j] = 1;
    std::vector<int> row_of(npos + 1, 0), slots;
    for (int p = 0; p < npos; p++) {
        row_of[p] = static_cast<int>(slots.size());
        if (needed[p]) slots.push_back(in.pos[p]);
    }
    row_of[npos] = static_cast<int>(slots.size());
    const int reg_row = reg_pos >= 0 ? row_of[reg_pos] : 0;
    const int nrows = out->rows = static_cast<int>(slots.size());
    // the last row each sub-batch reads
    int last_row[kHistMaxSub] = {0};
    for (int b = 0; b < nsub; b++) {
        if (b > 0 || !x_buffers) last_row[b] = reg_row + (b + 1) * nreg;
        for (int i = 0; i < ntau; i++)
            if (mask[static_cast<size_t>(b) * ntau + i])
                last_row[b] = std::max(last_row[b], row_of[in.ent_w[i] + b * nreg] + nreg);
        if (b > 0) last_row[b] = std::max(last_row[b], last_row[b - 1]);
    }
    // copies: pieces of consecutive ring slots inside a slab
    struct Piece {
        int slot, rows, row, stage;
    };
    std::vector<Piece> pieces, xpieces;
    auto cut = [](const int *slot, int n, std::vector<Piece> *out_pieces) {
        for (int u = 0; u < n;) {
            if (slot[u] < 0) {
                u++;
                continue;
            }
            if (slot[u] > 0xFFFFF) return false;
            int len = 1;
            while (u + len < n && slot[u + len] == slot[u] + len && (slot[u] + len) % kSlab != 0) len++;
            out_pieces->push_back(Piece{slot[u], len, u, 0});
            u += len;
        }
        return true;
    };
    if (!cut(slots.data(), nrows, &pieces) || (x_buffers && !cut(in.reg.data(), nreg, &xpieces)))
        return "ring slot index too large for a lag piece";
    const int npiece = static_cast<int>(pieces.size()), nx = static_cast<int>(xpieces.size());
    if (nrows > 0xFFFF) return "too many pieces for the resident-history lag kernel";
    // stages: sub-batch 0's pieces cut evenly, then one stage per further sub-batch
    int sub_stages[kHistMaxSub] = {0}, bytes[kHistStages] = {0}, x_bytes = 0;
    {
        int p0 = 0;
        while (p0 < npiece && pieces[p0].row < last_row[0]) p0++;
        const int parts = x_buffers ? std::min(kHistFirstStages, std::max(1, p0)) : 1;
        for (int i = 0; i < p0; i++) pieces[i].stage = i * parts / p0;
        sub_stages[0] = parts;
        int p = p0;
        for (int b = 1; b < nsub; b++) {
            for (; p < npiece && (b == nsub - 1 || pieces[p].row < last_row[b]); p++) pieces[p].stage = parts + b - 1;
            sub_stages[b] = parts + b;
        }
        for (; p < npiece; p++) pieces[p].stage = sub_stages[nsub - 1] - 1;
        for (const Piece &q : pieces) bytes[q.stage] += q.rows * kHistRowBytes;
        for (const Piece &q : xpieces) x_bytes += q.rows * kHistRowBytes;
    }
    // stages that hold the first `rows` rows; stages whose rows all lie below `row`
    auto stages_of = [&](int rows) {
        int st = 0;
        for (const Piece &q : pieces)
            if (q.row < rows) st = std::max(st, q.stage + 1);
        return st;
    };
    auto stages_below = [&](int row) {
        int st = sub_stages[nsub - 1];
        for (const Piece &q : pieces)
            if (q.row + q.rows > row) st = std::min(st, q.stage);
        return st;
    };
    out->frames = 0;
    for (const Piece &q : pieces) out->frames += q.rows;
    for (int j = 0; j < nreg && x_buffers; j++)  // register frames that no window holds
        out->frames += in.reg[j] >= 0 && (reg_pos < 0 || !needed[reg_pos + j]);
    int variants = 1;
    for (int b = 1; b < nsub; b++)
        for (int i = 0; i < ntau; i++) {
            const int m0 = mask[i], mb = mask[static_cast<size_t>(b) * ntau + i];
            if (m0 != mb || (mb && row_of[in.ent_w[i] + b * nreg] - b * nreg != row_of[in.ent_w[i]])) variants = nsub;
        }
    // units per sub-batch, put side by side for the half-warps and dealt to the warps
    const int halves = hist_halves(EB);
    std::vector<int> lptr;
    std::vector<HistStep> steps;
    auto build_variant = [&](int b) -> std::string {
        const int *mk = mask.data() + static_cast<size_t>(b) * ntau;
        std::vector<HistUnit> units[3];
        for (int i = 0; i < ntau;) {
            bool run = nreg == J && i + kLagFuse <= ntau;
            for (int r = 0; r < kLagFuse && run; r++) run = mk[i + r] == all && in.ent_w[i + r] == in.ent_w[i] + r;
            const int row = row_of[in.ent_w[i] + b * nreg] - b * nreg;
            if (run) {
                const int step = in.ent_acc[i + 1] - in.ent_acc[i];
                for (int r = 2; r < kLagFuse; r++)
                    if (in.ent_acc[i + r] != in.ent_acc[i] + r * step) return "accumulator rows of a fused run are not evenly spaced";
                units[kHistRun].push_back(HistUnit{kHistRun, row, in.ent_acc[i], step});
                i += kLagFuse;
            } else {
                const int kind = nreg == J && mk[i] == all ? kHistFull : kHistMasked;
                if (mk[i]) units[kind].push_back(HistUnit{kind, row, in.ent_acc[i], mk[i]});
                i++;
            }
        }
        struct Paired {
            HistUnit u[2];
            bool both;
        };
        std::vector<Paired> paired;
        for (int kind : {kHistRun, kHistMasked, kHistFull}) {  // by falling cost
            const auto &v = units[kind];
            for (size_t i = 0; i < v.size(); i += halves)
                paired.push_back(Paired{{v[i], v[std::min(i + halves - 1, v.size() - 1)]}, i + halves <= v.size()});
        }
        // longest first, each to the warp with the least work; a warp's steps in window order
        std::vector<std::vector<Paired>> list(CW);
        std::vector<double> load(CW, 0.0);
        for (const Paired &p : paired) {
            const int l = static_cast<int>(std::min_element(load.begin(), load.end()) - load.begin());
            list[l].push_back(p);
            load[l] += p.u[0].cost();
        }
        for (auto &l : list) {
            std::stable_sort(l.begin(), l.end(), [](const Paired &a, const Paired &c) { return a.u[0].row < c.u[0].row; });
            lptr.push_back(static_cast<int>(steps.size()) / halves);
            for (size_t s = 0; s < l.size(); s++)
                for (int h = 0; h < halves; h++) {
                    const HistUnit &u = l[s].u[h], &top = l[s].u[halves - 1];
                    // stages no unit from this step on reads (in the last sub-batch; a pair's first unit is its lowest)
                    const int below = stages_below(l[s].u[0].row + (nsub - 1) * nreg);
                    // stages for the step's rows (in a shared variant of later sub-batches all are there)
                    const int need = stages_of(top.row + (variants > 1 ? b : 0) * nreg + nreg +
                                               (u.kind == kHistRun ? kLagFuse - 1 : 0));
                    const bool active = h == 0 || l[s].both;
                    const int mask = u.kind == kHistRun ? u.mask * kHistRowBytes : u.mask;
                    steps.push_back(HistStep{u.row * kHistRowBytes, u.acc * kHistRowBytes, mask,
                                             u.kind | (active ? kHistActive : 0) | need << kHistNeedShift | below << kHistRelShift});
                }
        }
        return std::string();
    };
    for (int b = 0; b < variants; b++) {
        std::string err = build_variant(b);
        if (!err.empty()) return err;
    }
    lptr.push_back(static_cast<int>(steps.size()) / halves);
    const int head = kHtHeader + 2 * (npiece + nx) + static_cast<int>(lptr.size());
    const int steps_at = (head + 3) / 4 * 4;
    const size_t table_bytes = sizeof(int) * (steps_at + 4 * steps.size());
    out->smem = hist_table_offset(EB, buffers, nrows, nx) + table_bytes;
    if (out->smem > static_cast<size_t>(kHistSmemMax))
        return "the launch's frames do not fit in shared memory";
    out->ints.assign(steps_at + 4 * steps.size(), 0);
    int *t = out->ints.data();
    t[kHtNreg] = nreg;
    t[kHtNsub] = nsub;
    t[kHtNrows] = nrows;
    t[kHtNpiece] = npiece;
    t[kHtNx] = nx;
    t[kHtRegRow] = reg_row;
    t[kHtVariants] = variants;
    t[kHtBuffers] = buffers;
    t[kHtSteps] = steps_at;
    t[kHtInts] = static_cast<int>(out->ints.size());
    std::copy(sub_stages, sub_stages + kHistMaxSub, t + kHtSubStages);
    std::copy(bytes, bytes + kHistStages, t + kHtBytes);
    t[kHtXBytes] = x_bytes;
    t[kHtArrive] = 1;
    int *p = t + kHtHeader;
    for (const auto *v : {&pieces, &xpieces})
        for (const Piece &q : *v) {
            *p++ = q.slot | (q.rows - 1) << 20;
            *p++ = q.row | q.stage << 16;
        }
    std::copy(lptr.begin(), lptr.end(), p);
    if (!steps.empty()) std::memcpy(t + steps_at, steps.data(), sizeof(HistStep) * steps.size());
    out->steps = static_cast<int>(steps.size());
    return std::string();
}

// Upper bound of a table's ints for ntau entries over resident rows in `pieces` pieces (as many as
// rows at worst) and nsub sub-batches: every entry a unit of its own in every sub-batch, which is
// what launches without fused runs take.
inline int hist_table_capacity(int ntau, int pieces, int nsub) {
    return kHtHeader + 2 * (pieces + kHistMaxJ) + nsub * 12 + 1 + 3 + 4 * nsub * (ntau + 3);
}

// How an engine's launches run: elements per block, consumer warps per CTA, row buffers, and
// whether the register frames have buffers of their own.
struct HistShape {
    int EB = 0, CW = 0;  // 0: the launches do not fit and the ring kernel runs
    int buffers = 1;
    bool x_buffers = true;
};

// The table of a launch in the engine's shape. (A launch whose frames lie scattered over the ring
// may need more shared memory than the shape's CTAs per SM leave; it runs with fewer of them, or, if
// no CTA can hold it, without the register-frame buffers or with one row buffer.)
inline std::string build_hist_table(const HistInput &in, const HistShape &shape, HistTable *out) {
    std::string err = build_hist_table(in, shape.EB, shape.CW, shape.buffers, shape.x_buffers, out);
    if (!err.empty()) err = build_hist_table(in, shape.EB, shape.CW, 1, false, out);
    if (!err.empty()) err = build_hist_table(in, shape.EB, shape.CW, 1, true, out);
    return err;
}

// A full launch of an engine once every partner is there: its windows, in ring slots 0, 1, ... Compat:
// the windows start at the register frames and reach forward, else they reach back.
inline HistInput hist_steady(const std::vector<int> &taus, int batch, int nsub, int R, bool compat) {
    HistInput in;
    const int T = static_cast<int>(taus.size()), tau_max = taus.back();
    in.nreg = batch;
    in.nsub = nsub;
    for (int p = 0; p < tau_max + nsub * batch; p++) in.pos.push_back(p % R);
    for (int i = 0; i < T; i++) {
        in.ent_acc.push_back(i);
        in.ent_w.push_back(compat ? taus[i] : tau_max - taus[T - 1 - i]);
    }
    const int first = compat ? 0 : tau_max;
    in.reg.assign(in.pos.begin() + first, in.pos.begin() + first + nsub * batch);
    return in;
}

// Whether every launch with no more frames than `steady` fits a CTA of the shape, in one of the forms
// build_hist_table falls back to: no launch has other rows than the steady one, but its table may be
// several times as large (no fused runs without an instance for its frame count or with a partner
// missing; a list per sub-batch). Its pieces start at a window that does not touch the one before it,
// at the register frames, at the first frame there is, or at a slab's or the ring's first slot; with
// `scattered` positions (compat schedules) anywhere.
inline bool hist_always_fits(const HistInput &steady, const HistShape &shape, bool scattered) {
    const int ntau = static_cast<int>(steady.ent_acc.size());
    int starts = static_cast<int>(steady.pos.size()) / kSlab + 6;
    for (int i = 1; i < ntau; i++) starts += steady.ent_w[i] > steady.ent_w[i - 1] + 1;
    for (const bool x_buffers : {false, true}) {
        HistTable t;
        build_hist_table(steady, shape.EB, shape.CW, 1, x_buffers, &t);  // for its rows, whether it fits or not
        if (t.rows == 0) continue;
        const int ints = hist_table_capacity(ntau, scattered ? t.rows : std::min(t.rows, starts), steady.nsub);
        if (hist_table_offset(shape.EB, 1, t.rows, x_buffers) + sizeof(int) * ints <= static_cast<size_t>(kHistSmemMax))
            return true;
    }
    return false;
}

// Whether lags below 40 of very large frames in one or two scales are left to the ring kernel: its launches
// take no more time there, and the FFT writes whole frames faster than slabs (192 frames of 2048^2, two
// scales, ring kernel / this: 16 taus up to 28 12.0 ms / 13.3, 20 up to 20 12.0 / 13.1, 12 up to 32 11.8 / 12.7,
// 24 up to 32 13.4 / 14.1; 24 up to 40 14.9 / 14.1). With more scales the FFT's share is smaller (four, 12 up to 20
// 21.7 / 21.3; six, 14 up to 22 33.1 / 31.8), and smaller frames go either way by a few percent (1024^2, four
// scales, 20 up to 20 5.6 / 5.8, up to 30 5.6 / 5.4; 512^2, four, 12 up to 20 1374 us / 1257). Not where a chunk
// ends in a launch of a frame count without an instance, which the ring kernel runs masked (chunks of 25:
// 12.4 ms / 10.6).
inline bool hist_leave_to_ring(long long E, int scales, int tau_max, int chunk) {
    constexpr long long kMinElements = 1LL << 22;
    const int rest = chunk < kHistMaxJ ? chunk : chunk % kHistMaxJ;
    return E >= kMinElements && scales <= 2 && tau_max < 40 && (rest == 0 || hist_pick_j(rest) == rest);
}

// Dynamic shared memory a launch asks for, given what its table needs. Three CTAs of up to 54 KB take the
// same split of an SM's memory as the FFT passes' CTAs (164 KB), and the next piece's FFT, queued at the
// same time, then mixes with a lag launch that needs all of its CTAs at once. For frames of up to 512^2 the two
// took longer than one after the other (192 frames in submits of 32, 512^2, four scales: 24 taus up to 600
// 3213 us, with 56,000 bytes 2504, ring kernel 2558; 64 up to 300 3030 / 2855; 20 up to 1000 2622 / 2488;
// two scales: 1709 / 1542, 1410 / 1348, 1404 / 1334). Larger frames measured the same either way (1024^2, one
// to four scales: within 1 %), small launches gain from the mixing (256^2, three scales: 3 - 4 %; 512^2, one: 1 %).
inline size_t hist_launch_smem(size_t table_smem, int side, long long E) {
    constexpr size_t kOwnSplit = 56000;
    constexpr long long kMinElements = 200000;
    return side <= 512 && E >= kMinElements ? std::max(table_smem, kOwnSplit) : table_smem;
}

// The shape for launches like `steady` (every partner there): as many CTAs per SM as the rows
// leave room for, with the widest block (a thread of a wider block walks more entries per load of
// its register frames), and in their shared memory whole blocks in two or more row buffers, else
// one buffer with register-frame buffers. One buffer alone (a block then starts only when all its
// rows are there) comes after the narrower block: 32-frame launches of 512^2, four scales, 64 taus
// up to 300, took 569 us with it, 514 in the ring kernel and 430 with blocks of 16 and
// register-frame buffers. The ring kernel keeps short tau lists, whose blocks are too little work for
// their barriers (192 frames in submits of 32, with the FFT, per 32, ring kernel / this: 1024^2, four scales, 6 taus
// up to 20 756 us / 800, up to 100 867 / 849, 8 up to 20 791 / 809, up to 100 925 / 885, up to 300 1006 / 1068, 10 up
// to 100 961 / 919; 512^2, four scales, 6 up to 20 154 / 162, 8 up to 20 161 / 164, up to 100 190 / 186), and those
// that one CTA per SM would run without many taus: its one row buffer is loaded for little work (192 frames of 512^2, two scales, submits of 32,
// ring kernel / this: 100 taus up to 1300 3247 us / 3640, 80 up to 1650 2930 / 3600; 128 up to 1000 3550 / 3407,
// up to 1300 4320 / 3614). Launches of two batches save more reads (against single batches: 48 up to 1300
// 1997 / 2416, 64 up to 1000 2110 / 2427, 80 2256 / 2517; 100 up to 1000 2817 / 2648, 128 3407 / 2676).
// A shape is taken only if no launch of the engine can outgrow it (hist_always_fits): the ring's
// layout follows the kernel, so there is no other one to go to later.
inline HistShape hist_pick_shape(const HistInput &steady, bool scattered) {
    constexpr int kMinTaus = 8;
    const int kMinTausOneCta = steady.nsub > 1 ? 96 : 112;
    const struct {
        int EB, CW, taus;
        bool bare;
    } sizes[] = {{32, 4, kMinTaus, false}, {16, 4, kMinTaus, true}, {16, 6, kMinTaus, true}, {16, 12, kMinTausOneCta, true}};
    HistTable t;
    for (const auto &size : sizes) {
        if (static_cast<int>(steady.ent_acc.size()) < size.taus) continue;
        HistShape s;
        s.EB = size.EB;
        s.CW = size.CW;
        auto fits = [&](int buffers, bool x_buffers) {
            s.buffers = buffers;
            s.x_buffers = x_buffers;
            return build_hist_table(steady, s.EB, s.CW, buffers, x_buffers, &t).empty() &&
                   t.smem <= static_cast<size_t>(hist_smem_limit(s.CW));
        };
        bool found = false;
        for (int buffers = kHistMaxBuffers; buffers >= 2 && !found; buffers--) found = fits(buffers, false);
        found = found || fits(1, true) || (size.bare && fits(1, false));
        if (found && hist_always_fits(steady, s, scattered)) return s;
    }
    return HistShape();
}

}  // namespace ddm
