// Planning of fused passes: the scan that groups one- and two-axis operations
// into passes (and a pass's operations into register rounds), and the
// descriptors and coefficients of the CUDA-core passes.
//
// The scan.  Operations on disjoint axes commute, so an operation may run in
// an earlier pass than one that precedes it in program order, provided every
// earlier operation sharing one of its axes has run.  For each pass the
// pending operations are scanned in order; an operation is taken when its
// axes fit beside the resident ones and none of them is held back by an
// operation that could not be taken, otherwise its own axes are held back.
// A scan ends early once nothing later can be taken.  Successive one-axis
// maps on one axis take the same slot: they are multiplied into one map.
//
// Axis sets are bit masks and the pending operations one index list that is
// compacted per pass.  In the interpreter the same scan over sets of axes and
// one descriptor field at a time took most of a small circuit's host time: a
// call with 20 noisy layers on 8 qubits (558 operations, 13 FP64 passes) took
// 6.7 ms end to end with it, 3.8 ms with this file.
// Host code only; no CUDA.
#include <stdint.h>
#include <string.h>

#include <exception>
#include <vector>

#include "dm_gb300.h"

namespace {

inline int popcount(uint32_t x) { return __builtin_popcount(x); }

inline uint32_t axis_mask(const dm_plan_op &op) {
    return (1u << op.a) | (op.kind == DM_OP_MAP1 ? 0u : 1u << op.b);
}

inline int coefficients(int32_t kind) {
    return kind == DM_OP_CX ? 5 : kind == DM_OP_MAP2 ? 256 : 16;
}

// Assign ops to passes over n axes of at most kmax resident ones, `base` always resident.
// pass_of[i] = -1 where partial planning leaves op i.  False when an op fits no pass.
bool scan(const dm_plan_op *ops, int count, int n, int kmax, uint32_t base, bool partial, int32_t *pass_of,
          int32_t *slot_of, std::vector<uint32_t> &resident_of) {
    std::vector<int32_t> pending(static_cast<size_t>(count));
    for (int i = 0; i < count; ++i) {
        pending[size_t(i)] = i;
        pass_of[i] = -1;
        slot_of[i] = -1;
    }
    std::vector<int32_t> left;
    while (!pending.empty()) {
        const int32_t pass = int32_t(resident_of.size());
        uint32_t resident = base, blocked = 0;
        int taken = 0, slots = 0;
        int32_t last[32];              // slot of the last op on an axis, negative: none, or a pair op
        for (int a = 0; a < 32; ++a) last[a] = -1;
        bool closed = false;
        size_t i = 0;
        left.clear();
        for (; i < pending.size(); ++i) {
            const dm_plan_op &op = ops[pending[i]];
            const uint32_t m = axis_mask(op);
            if ((blocked & m) || popcount(resident | m) > kmax || slots >= DM_MAX_PASS_OPS) {
                blocked |= m;
                left.push_back(pending[i]);
                if ((popcount(resident) >= kmax && (resident & ~blocked) == 0) || popcount(blocked) >= n) {
                    closed = true;
                    ++i;
                    break;
                }
                continue;
            }
            resident |= m;
            ++taken;
            pass_of[pending[i]] = pass;
            if (op.kind == DM_OP_MAP1) {
                if (last[op.a] < 0) last[op.a] = slots++;
                slot_of[pending[i]] = last[op.a];
            } else {
                slot_of[pending[i]] = slots++;
                last[op.a] = last[op.b] = -1;
            }
        }
        if (!taken) return false;
        if (partial && !closed) {      // later ops could still join this pass
            for (size_t j = 0; j < pending.size(); ++j) pass_of[pending[j]] = slot_of[pending[j]] = -1;
            return true;
        }
        left.insert(left.end(), pending.begin() + int64_t(i), pending.end());
        pending.swap(left);
        resident_of.push_back(resident);
    }
    return true;
}

bool valid(const dm_plan_op *ops, int count, int n) {
    for (int i = 0; i < count; ++i) {
        if (ops[i].kind < DM_OP_MAP1 || ops[i].kind > DM_OP_CX) return false;
        if (ops[i].a < 0 || ops[i].a >= n) return false;
        if (ops[i].kind != DM_OP_MAP1 && (ops[i].b < 0 || ops[i].b >= n || ops[i].a == ops[i].b)) return false;
    }
    return true;
}

// c = a b for 4x4 maps
void multiply(const double *a, const double *b, double *c) {
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j) {
            double s = 0.0;
            for (int k = 0; k < 4; ++k) s += a[4 * i + k] * b[4 * k + j];
            c[4 * i + j] = s;
        }
}

struct Composed {
    dm_plan_op op;                     // axes: local to the pass
    const double *data;
};

// Group the ops of one pass or round by slot; maps that share a slot are multiplied in order.  False where
// the slots are not what a scan gives: taken in order, and shared by one-axis maps on one axis only (a slot
// shared by a CX would read its 5 coefficients as 16).
bool compose(const dm_plan_op *ops, const double *const *data, const std::vector<int32_t> &members,
             const int32_t *slot_of, std::vector<Composed> &body, std::vector<double> &products) {
    body.clear();
    products.clear();
    products.reserve(16 * members.size());       // pointers into it stay valid
    for (const int32_t i : members) {
        const size_t slot = size_t(slot_of[i]);
        if (slot < body.size()) {
            const dm_plan_op &first = body[slot].op;
            if (first.kind != DM_OP_MAP1 || ops[i].kind != DM_OP_MAP1 || first.a != ops[i].a) return false;
            double c[16];
            multiply(data[i], body[slot].data, c);
            const size_t at = products.size();
            products.insert(products.end(), c, c + 16);
            body[slot].data = products.data() + at;
        } else {
            if (slot != body.size()) return false;
            body.push_back({ops[i], data[i]});
        }
    }
    return true;
}

int plan(int n, int kmax, int low, const dm_plan_op *ops, int count, int partial, int32_t *pass_of, int32_t *slot_of,
         uint32_t *resident, int32_t *npasses) {
    if (n < 1 || n > 30 || kmax < 0 || low < 0 || count < 0 || !npasses) return DM_ERR_ARG;
    if (count > 0 && (!ops || !pass_of || !slot_of || !resident)) return DM_ERR_ARG;
    if (!valid(ops, count, n)) return DM_ERR_ARG;
    if (kmax > n) kmax = n;
    if (low > kmax) low = kmax;
    const uint32_t base = ((1u << low) - 1u) << (n - low);
    std::vector<uint32_t> masks;
    if (!scan(ops, count, n, kmax, base, partial != 0, pass_of, slot_of, masks)) return DM_ERR_PROGRAM;
    *npasses = int32_t(masks.size());
    if (!masks.empty()) memcpy(resident, masks.data(), masks.size() * sizeof(uint32_t));
    return DM_OK;
}

int encode(int n, int dtype, int width, int max_axes, const dm_plan_op *ops, int count, const double *coefs,
           const int32_t *pass_of, const int32_t *slot_of, const uint32_t *resident, int npasses, size_t mats_off,
           dm_pass *passes, void *mats, size_t mats_capacity, size_t *mats_used) {
    if (n < 1 || n > 30 || (dtype != DM_F32 && dtype != DM_F64) || count < 0 || npasses < 0 || !mats_used ||
        width < 0 || width > 4)
        return DM_ERR_ARG;
    if (npasses > 0 && (!ops || !coefs || !pass_of || !slot_of || !resident || !passes || !mats)) return DM_ERR_ARG;
    if (!valid(ops, count, n)) return DM_ERR_ARG;
    std::vector<const double *> data(static_cast<size_t>(count));
    std::vector<std::vector<int32_t>> members(static_cast<size_t>(npasses));
    for (int i = 0; i < count; ++i) {
        data[size_t(i)] = coefs;
        coefs += coefficients(ops[i].kind);
        if (pass_of[i] < 0) continue;
        if (pass_of[i] >= npasses || slot_of[i] < 0 || slot_of[i] >= DM_MAX_PASS_OPS) return DM_ERR_ARG;
        members[size_t(pass_of[i])].push_back(i);
    }
    size_t used = 0;
    std::vector<Composed> body, regrouped;
    std::vector<double> products, round_products;
    std::vector<dm_plan_op> local;
    std::vector<const double *> local_data;
    for (int p = 0; p < npasses; ++p) {
        dm_pass &dp = passes[p];
        memset(&dp, 0, sizeof(dp));
        int local_of[32];
        dp.k = 0;
        for (int q = n - 1; q >= 0; --q)
            if (resident[p] >> q & 1) {
                if (dp.k == DM_MAX_TILE_AXES) return DM_ERR_ARG;
                local_of[q] = dp.k;
                dp.axes[dp.k++] = q;
            }
        if (!compose(ops, data.data(), members[size_t(p)], slot_of, body, products) || body.size() > DM_MAX_PASS_OPS)
            return DM_ERR_ARG;
        bool map2 = false;
        local.clear();
        local_data.clear();
        for (Composed &c : body) {
            if (!(resident[p] >> c.op.a & 1) || (c.op.kind != DM_OP_MAP1 && !(resident[p] >> c.op.b & 1)))
                return DM_ERR_ARG;
            c.op.a = int16_t(local_of[c.op.a]);
            c.op.b = c.op.kind == DM_OP_MAP1 ? int16_t(0) : int16_t(local_of[c.op.b]);
            map2 = map2 || c.op.kind == DM_OP_MAP2;
            local.push_back(c.op);
            local_data.push_back(c.data);
        }
        // register rounds: the same scan over the pass's own axes
        std::vector<int32_t> round_of(local.size()), round_slot(local.size());
        std::vector<uint32_t> round_axes;
        bool rounds = width > 0 && width <= dp.k && dp.k <= max_axes && dp.axes[0] == n - 1 && !map2;
        if (rounds && !scan(local.data(), int(local.size()), dp.k, width, 0, false, round_of.data(), round_slot.data(),
                            round_axes))
            return DM_ERR_PROGRAM;
        rounds = rounds && round_axes.size() <= DM_MAX_ROUNDS;
        auto emit = [&](const Composed &c, int32_t digits) {
            dm_op &o = dp.ops[dp.nops++];
            const int len = coefficients(c.op.kind);
            if (used + size_t(len) > mats_capacity) return false;
            const double *m = c.data;
            o.kind = c.op.kind;
            o.a = c.op.a;
            o.b = c.op.b;
            o.moff = int32_t(mats_off + used);
            o.flags = digits;
            if (c.op.kind == DM_OP_MAP1) {
                if (m[0] == 1.0 && m[1] == 0.0 && m[2] == 0.0 && m[3] == 0.0) o.flags |= DM_MAP1_ROW0_IDENTITY;
                if (m[4] == 0.0 && m[8] == 0.0) o.flags |= DM_MAP1_XY_UNITAL;
            } else if (c.op.kind == DM_OP_CX && c.op.ideal) {
                o.flags |= DM_CX_IDEAL;
            }
            if (dtype == DM_F64)
                memcpy(static_cast<double *>(mats) + used, m, size_t(len) * sizeof(double));
            else
                for (int j = 0; j < len; ++j) static_cast<float *>(mats)[used + size_t(j)] = float(m[j]);
            used += size_t(len);
            return true;
        };
        if (!rounds) {
            for (const Composed &c : body)
                if (!emit(c, 0)) return DM_ERR_ARG;
            continue;
        }
        dp.nrounds = int32_t(round_axes.size());
        std::vector<std::vector<int32_t>> by_round(round_axes.size());
        for (size_t i = 0; i < local.size(); ++i) by_round[size_t(round_of[i])].push_back(int32_t(i));
        for (size_t r = 0; r < round_axes.size(); ++r) {
            uint32_t axes = round_axes[r];
            // padded with the lowest axes: axis 0 in a round lets the kernel move 16-byte vectors
            for (int a = 0; popcount(axes) < width; ++a) axes |= 1u << a;
            int at[32], d = 0;
            for (int a = 0; a < dp.k; ++a)
                if (axes >> a & 1) {
                    at[a] = d;
                    dp.round_axes[r][d++] = int8_t(a);
                }
            for (; d < 4; ++d) dp.round_axes[r][d] = -1;
            if (!compose(local.data(), local_data.data(), by_round[r], round_slot.data(), regrouped, round_products))
                return DM_ERR_PROGRAM;
            for (const Composed &c : regrouped) {
                const int32_t digits = (at[c.op.a] << 8) | (c.op.kind == DM_OP_MAP1 ? 0 : at[c.op.b] << 12);
                if (!emit(c, digits)) return DM_ERR_ARG;
            }
            dp.round_end[r] = int16_t(dp.nops);
        }
    }
    *mats_used = used;
    return DM_OK;
}

// No exception leaves the C entry points: what the standard library throws is memory it did not get.
template <typename F>
int guarded(F f) {
    try {
        return f();
    } catch (const std::exception &) {
        return DM_ERR_MEMORY;
    }
}

}  // namespace

extern "C" int dm_plan_passes(int n, int kmax, int low, const dm_plan_op *ops, int count, int partial,
                              int32_t *pass_of, int32_t *slot_of, uint32_t *resident, int32_t *npasses) {
    return guarded([&] { return plan(n, kmax, low, ops, count, partial, pass_of, slot_of, resident, npasses); });
}

extern "C" int dm_encode_passes(int n, int dtype, int width, int max_axes, const dm_plan_op *ops, int count,
                                const double *coefs, const int32_t *pass_of, const int32_t *slot_of,
                                const uint32_t *resident, int npasses, size_t mats_off, dm_pass *passes, void *mats,
                                size_t mats_capacity, size_t *mats_used) {
    return guarded([&] {
        return encode(n, dtype, width, max_axes, ops, count, coefs, pass_of, slot_of, resident, npasses, mats_off, passes,
                      mats, mats_capacity, mats_used);
    });
}
