// Matching of recorded dispatches with fused launches (fuse.h). A dispatch may join one recorded before it when nothing
// recorded in between touches any range it binds (reads of the same range count as touching: the check knows no directions),
// so running it early changes neither what it reads nor what the others read. Only kernels whose effects are confined to
// their bindings are looked past (the output exchange between ranks and kernels a host has registered are not). A form is
// taken only when every member, and every dispatch it is moved past, passes the checks of its own launcher; anything else is
// launched by itself, errors included: when a dispatch is refused, nothing recorded behind it has run.
#include "fuse.h"

namespace amv {

AcResult launch_add_f32(const LaunchArgs&);
AcResult launch_bitnet_gemm_i2_s(const LaunchArgs&);
AcResult launch_bitnet_gemv_i2_s(const LaunchArgs&);
AcResult launch_bitnet_norm_q8(const LaunchArgs&);
AcResult launch_mmvq_q4_1(const LaunchArgs&);
AcResult launch_mmvqb_iq4_xs(const LaunchArgs&);
AcResult launch_mmvqb_q2_K(const LaunchArgs&);
AcResult launch_mmvqb_q3_K(const LaunchArgs&);
AcResult launch_mmvqb_q5_K(const LaunchArgs&);
AcResult launch_mmvqb_q6_K(const LaunchArgs&);
AcResult launch_quant_a8(const LaunchArgs&);
AcResult launch_quant_a8_f16(const LaunchArgs&);
AcResult launch_quant_a8b(const LaunchArgs&);
AcResult launch_quant_a8b_f16(const LaunchArgs&);
AcResult launch_rms_norm_f32(const LaunchArgs&);
AcResult launch_rms_norm_quant_a8(const LaunchArgs&);
AcResult launch_rms_norm_quant_a8b(const LaunchArgs&);
AcResult launch_rope(const LaunchArgs&);
AcResult launch_set_rows(const LaunchArgs&);
AcResult launch_swiglu_f32(const LaunchArgs&);

namespace {

constexpr uint32_t kLookahead = 12;   // operations looked at past the first

bool is(const FuseOp& op, LaunchFn fn) { return op.entry->launch == fn; }

bool overlap(const void* p, uint64_t n, const void* q, uint64_t m) {
    const uintptr_t a = (uintptr_t)p, b = (uintptr_t)q;
    return a < b + m && b < a + n;
}
bool touches(const LaunchArgs& a, const void* p, uint64_t n) {
    for (uint32_t i = 0; i < a.binding_count; ++i)
        if (overlap(a.ptr[i], a.range[i], p, n)) return true;
    return false;
}
bool disjoint(const LaunchArgs& a, const LaunchArgs& b) {
    for (uint32_t i = 0; i < b.binding_count; ++i)
        if (touches(a, b.ptr[i], b.range[i])) return false;
    return true;
}

// kernels that read and write their bindings and nothing else (products without the exchange between ranks, quantizes)
bool starts(const FuseOp& op, const char* prefix) { return strncmp(op.entry->name, prefix, strlen(prefix)) == 0; }
bool confined(const FuseOp& op) {
    if (!op.entry->launch) return false;
    if (starts(op, "ameva_mmvs_")) return op.args.push[4] == 0u;   // (peers)
    return is(op, launch_bitnet_gemv_i2_s) || is(op, launch_bitnet_gemm_i2_s) || is(op, launch_bitnet_norm_q8) ||
           starts(op, "ameva_quant_a8") || ((starts(op, "ameva_mmv") || starts(op, "ameva_mmtc_")) && !strstr(op.entry->name, "_mp"));
}

// May ops[j] run together with ops[i], i < j? Members of the group being formed (marked in `member`) are checked by the caller.
bool can_hoist(FuseOp* ops, uint32_t i, uint32_t j, uint64_t member) {
    for (uint32_t k = i + 1; k < j; ++k) {
        if (ops[k].done || (member >> (k - i) & 1u)) continue;
        if (!confined(ops[k]) || !disjoint(ops[k].args, ops[j].args)) return false;
        if (ops[k].checks == FuseOp::UNKNOWN) {
            LaunchArgs a = ops[k].args;
            a.stream.dry = true;
            ops[k].checks = ops[k].entry->launch(a) == AC_SUCCESS ? FuseOp::PASSES : FuseOp::REFUSED;
        }
        if (ops[k].checks == FuseOp::REFUSED) return false;
    }
    return true;
}

// ---- RMS norm, SWIGLU or nothing, then the quantize of every I2_S product that reads the rows ----
AcResult fuse_bitnet_rows(FuseOp* ops, uint32_t n, uint32_t i, bool* taken) {
    const LaunchArgs& head = ops[i].args;
    BitnetSource source = BITNET_PLAIN;
    const void* rows_ptr = head.ptr[0];
    uint32_t dim = 0, rows = 0;
    const LaunchArgs* member[kFuseMax];
    uint32_t count = 0;
    uint64_t mask = 0;
    if (is(ops[i], launch_bitnet_norm_q8)) {
        if (check_bitnet_norm_q8(head) != AC_SUCCESS || !bitnet_rows_fits(head)) return AC_SUCCESS;
        dim = head.push[0];
        rows = head.grid.x;
        member[count++] = &head;
    } else if (is(ops[i], launch_rms_norm_f32)) {
        source = BITNET_NORM;
        rows = head.push[0];
        dim = head.push[1];
        rows_ptr = head.ptr[2];
        float eps;
        memcpy(&eps, &head.push[2], 4);
        const uint64_t bytes = (uint64_t)rows * dim * 4u;
        if (!rows || !dim || head.push[3] > 1u || !(eps >= 0.0f) || head.range[0] < bytes || head.range[2] < bytes ||
            (head.push[3] && (head.range[1] < (uint64_t)dim * 4u || ((uintptr_t)head.ptr[1] & 15u) ||
                              overlap(head.ptr[1], (uint64_t)dim * 4u, head.ptr[2], bytes))))
            return AC_SUCCESS;
        if (head.ptr[0] != head.ptr[2] && overlap(head.ptr[0], bytes, head.ptr[2], bytes)) return AC_SUCCESS;
    } else {
        source = BITNET_SWIGLU;
        rows_ptr = head.ptr[2];
    }
    const uint64_t swiglu_n = source == BITNET_SWIGLU ? head.push[0] : 0u;
    for (uint32_t j = i + 1; j < n && j <= i + kLookahead && count < kFuseMax; ++j) {
        if (ops[j].done) continue;
        const LaunchArgs& q = ops[j].args;
        if (is(ops[j], launch_bitnet_norm_q8) && q.ptr[0] == rows_ptr && check_bitnet_norm_q8(q) == AC_SUCCESS && bitnet_rows_fits(q)) {
            bool ok = true;
            if (source == BITNET_SWIGLU && count == 0) {   // the first quantize says how the elements form rows
                dim = q.push[0];
                rows = q.grid.x;
                const uint64_t bytes = swiglu_n * 4u;
                ok = swiglu_n && (uint64_t)dim * rows == swiglu_n && head.range[0] >= bytes && head.range[1] >= bytes &&
                     head.range[2] >= bytes && (head.ptr[0] == head.ptr[2] || !overlap(head.ptr[0], bytes, head.ptr[2], bytes)) &&
                     (head.ptr[1] == head.ptr[2] || !overlap(head.ptr[1], bytes, head.ptr[2], bytes)) && !((uintptr_t)head.ptr[1] & 15u);
            }
            ok = ok && q.push[0] == dim && q.grid.x == rows && !((uintptr_t)head.ptr[0] & 15u) && can_hoist(ops, i, j, mask);
            // what this member writes (y, q, act, qeo) meets nothing that the head or another member reads or writes
            for (uint32_t b = 3; b < 7u && ok; ++b) {
                for (uint32_t h = 0; h < head.binding_count && ok; ++h) {
                    if (source == BITNET_NORM && h == 1u && !head.push[3]) continue;   // (the unused weight binding)
                    if (source == BITNET_PLAIN && (h == 1u || h == 2u)) continue;      // (b and w, unused in this mode)
                    ok = !overlap(head.ptr[h], head.range[h], q.ptr[b], q.range[b]);
                }
                for (uint32_t m = 0; m < count && ok; ++m)
                    for (uint32_t h = 3; h < 7u && ok; ++h) ok = !overlap(member[m]->ptr[h], member[m]->range[h], q.ptr[b], q.range[b]);
                for (uint32_t h = 3; h < b && ok; ++h) ok = !overlap(q.ptr[h], q.range[h], q.ptr[b], q.range[b]);
                ok = ok && !overlap(rows_ptr, (uint64_t)rows * dim * 4u, q.ptr[b], q.range[b]);
            }
            if (ok) {
                member[count++] = &q;
                mask |= 1ull << (j - i);
                continue;
            }
        }
        if (!confined(ops[j])) break;
    }
    if (count == 0 || (count == 1 && source == BITNET_PLAIN)) return AC_SUCCESS;
    if (rows > 0x7fffffffu) return AC_SUCCESS;
    *taken = true;
    ops[i].done = true;
    for (uint32_t k = 0; k <= kLookahead; ++k)
        if (mask >> k & 1u) ops[i + k].done = true;
    return launch_bitnet_rows(source, &head, member, count);
}

// ---- I2_S products: several in one launch, or one with the ADD that consumes it ----
AcResult fuse_bitnet_gemv(FuseOp* ops, uint32_t n, uint32_t i, bool* taken) {
    const LaunchArgs& head = ops[i].args;
    if (check_bitnet_gemv_i2_s(head) != AC_SUCCESS) return AC_SUCCESS;
    const uint32_t K = head.push[0], M = head.push[4] ? head.push[4] : 1u;
    const LaunchArgs* member[kFuseMax] = {&head};
    uint32_t count = 1;
    uint64_t mask = 0;
    for (uint32_t j = i + 1; j < n && j <= i + kLookahead && count < kFuseMax; ++j) {
        if (ops[j].done) continue;
        const LaunchArgs& p = ops[j].args;
        if (M <= 2u && is(ops[j], launch_bitnet_gemv_i2_s) && !p.stream.in_order && p.push[0] == K && (p.push[4] ? p.push[4] : 1u) == M &&
            check_bitnet_gemv_i2_s(p) == AC_SUCCESS && can_hoist(ops, i, j, mask)) {
            bool ok = true;   // no product writes what another one reads or writes
            for (uint32_t m = 0; m < count && ok; ++m)
                ok = !touches(*member[m], p.ptr[2], p.range[2]) && !touches(p, member[m]->ptr[2], member[m]->range[2]);
            if (ok) {
                member[count++] = &p;
                mask |= 1ull << (j - i);
                continue;
            }
        }
        if (!confined(ops[j])) break;
    }
    const LaunchArgs* add = nullptr;
    bool swapped = false;
    uint32_t add_at = 0;
    if (count == 1) {   // the next operation adds rows to the product
        uint32_t j = i + 1;
        while (j < n && ops[j].done) ++j;
        if (j < n && is(ops[j], launch_add_f32)) {
            const LaunchArgs& s = ops[j].args;
            const uint32_t N = head.push[1], stride = head.push[5] ? head.push[5] : N;
            const uint64_t bytes = (uint64_t)M * N * 4u;
            const char* product = (const char*)head.ptr[2] + 4ull * head.push[3];
            swapped = s.ptr[1] == product;
            const void* e = s.ptr[swapped ? 0 : 1];
            if ((swapped || s.ptr[0] == product) && stride == N && s.push[0] == M && s.push[1] == N && s.push[2] == M &&
                s.range[0] >= bytes && s.range[1] >= bytes && s.range[2] >= bytes && !overlap(e, bytes, product, bytes) &&
                (e == s.ptr[2] || !overlap(e, bytes, s.ptr[2], bytes)) && !touches(head, s.ptr[2], s.range[2])) {
                add = &s;
                add_at = j;
            }
        }
        if (!add) return AC_SUCCESS;
        ops[add_at].done = true;
    }
    *taken = true;
    ops[i].done = true;
    for (uint32_t k = 0; k <= kLookahead; ++k)
        if (mask >> k & 1u) ops[i + k].done = true;
    return launch_bitnet_gemv_i2_s_group(member, count, add, swapped);
}

// ---- a product of a byte-decoded type with the ADD that consumes it ----
AcResult fuse_product_add(FuseOp* ops, uint32_t n, uint32_t i, bool* taken) {
    LaunchArgs p = ops[i].args;
    const uint32_t M = p.push[0], N = p.push[1];
    uint32_t j = i + 1;
    while (j < n && ops[j].done) ++j;
    if (j >= n || !is(ops[j], launch_add_f32) || !M || !N || p.push[3] != N) return AC_SUCCESS;
    const LaunchArgs& s = ops[j].args;
    const uint64_t bytes = (uint64_t)M * N * 4u;
    const bool swapped = s.ptr[1] == p.ptr[4];
    void* e = s.ptr[swapped ? 0 : 1];
    if (!(swapped || s.ptr[0] == p.ptr[4]) || s.push[0] != M || s.push[1] != N || s.push[2] != M || s.range[0] < bytes ||
        s.range[1] < bytes || s.range[2] < bytes || overlap(e, bytes, p.ptr[4], bytes) ||
        (e != s.ptr[2] && overlap(e, bytes, s.ptr[2], bytes)) || touches(p, s.ptr[2], s.range[2]))
        return AC_SUCCESS;
    p.add_e = (const float*)e;
    p.add_out = (float*)s.ptr[2];
    *taken = true;
    ops[i].done = ops[j].done = true;
    return ops[i].entry->launch(p);
}

// ---- ROPEs and cache writes in a row ----
// Ranges an operation reads (ROPE: source, positions, factors; SET_ROWS: source, indices); both write binding 3. A status
// binding (SET_ROWS 2) takes atomics only, so several operations may share it.
bool row_op_writes_meet(const LaunchArgs& w, const LaunchArgs& other, bool other_rope, bool except_source) {
    for (uint32_t b = 0; b < 4u; ++b) {
        if (b == 0u && except_source) continue;
        if (b == 2u && other_rope && !other.push[16]) continue;   // (no frequency factors: the binding is not read)
        if (overlap(w.ptr[3], w.range[3], other.ptr[b], other.range[b])) return true;
    }
    return false;
}
bool status_meets(const LaunchArgs& set, const LaunchArgs& other, bool other_rope) {
    for (uint32_t b = 0; b < 4u; ++b)
        if ((b != 2u || (other_rope && other.push[16])) && overlap(set.ptr[2], set.range[2], other.ptr[b], other.range[b])) return true;
    return false;
}

AcResult fuse_row_ops(FuseOp* ops, uint32_t n, uint32_t i, bool* taken) {
    const LaunchArgs *rope[2], *store[2] = {nullptr, nullptr}, *set[2];
    uint32_t n_rope = 0, n_set = 0, count = 0, at[6];
    for (uint32_t j = i; j < n && count < 6u; ++j) {
        if (ops[j].done) continue;
        const bool r = is(ops[j], launch_rope);
        if (!r && !is(ops[j], launch_set_rows)) break;
        const LaunchArgs& p = ops[j].args;
        if (!row_op_serves(p, r)) break;
        int chain = -1;
        if (!r)
            for (uint32_t k = 0; k < n_rope; ++k)
                if (!store[k] && rope_feeds_set_rows(*rope[k], p)) chain = (int)k;
        if (r ? n_rope == 2u : (chain < 0 && n_set == 2u)) break;
        bool ok = true;
        for (uint32_t k = 0; k < count && ok; ++k) {
            const LaunchArgs& o = ops[at[k]].args;
            const bool o_rope = is(ops[at[k]], launch_rope), source = chain >= 0 && &o == rope[chain];
            // neither writes what the other reads or writes (the rotated rows that p stores excepted)
            ok = !row_op_writes_meet(p, o, o_rope, false) && !row_op_writes_meet(o, p, r, source) &&
                 (r || !status_meets(p, o, o_rope)) && (o_rope || !status_meets(o, p, r));
        }
        if (!ok) break;
        if (r) rope[n_rope++] = &p;
        else if (chain >= 0) store[chain] = &p;
        else set[n_set++] = &p;
        at[count++] = j;
    }
    if (count < 2u) return AC_SUCCESS;
    *taken = true;
    for (uint32_t k = 0; k < count; ++k) ops[at[k]].done = true;
    return launch_row_ops(ops[i].args.stream, rope, store, n_rope, set, n_set);
}

// ---- per-32 / per-256 quantizes of the same rows ----
bool quant_of(const FuseOp& op, QuantForm* form, uint32_t* scheme) {
    if (is(op, launch_quant_a8) || is(op, launch_quant_a8b)) *form = QUANT_PLAIN;
    else if (is(op, launch_quant_a8_f16) || is(op, launch_quant_a8b_f16)) *form = QUANT_F16;
    else if (is(op, launch_rms_norm_quant_a8) || is(op, launch_rms_norm_quant_a8b)) *form = QUANT_NORM;
    else return false;
    *scheme = is(op, launch_quant_a8b) || is(op, launch_quant_a8b_f16) || is(op, launch_rms_norm_quant_a8b);
    return true;
}

AcResult fuse_quant(FuseOp* ops, uint32_t n, uint32_t i, bool* taken) {
    const LaunchArgs& head = ops[i].args;
    const bool swiglu = is(ops[i], launch_swiglu_f32);
    QuantForm form = QUANT_PLAIN, want = QUANT_PLAIN;   // of the first quantize, and of those that may join it
    uint32_t scheme = 0, K = 0, M = 0;
    const LaunchArgs* first = nullptr;
    const void* rows_ptr = nullptr;
    uint64_t rows_bytes = 0;
    if (swiglu) {
        rows_ptr = head.ptr[2];
        rows_bytes = 4ull * head.push[0];
        if (!rows_bytes || head.range[0] < rows_bytes || head.range[1] < rows_bytes || head.range[2] < rows_bytes) return AC_SUCCESS;
        for (uint32_t b = 0; b < 2u; ++b)
            if (((uintptr_t)head.ptr[b] & 15u) || (head.ptr[b] != rows_ptr && overlap(head.ptr[b], rows_bytes, rows_ptr, rows_bytes)))
                return AC_SUCCESS;
    } else {
        quant_of(ops[i], &form, &scheme);
        if (check_quant(head, form, scheme) != AC_SUCCESS) return AC_SUCCESS;
        first = &head;
        M = head.push[0];
        K = head.push[1];
        rows_ptr = form == QUANT_NORM ? head.ptr[2] : head.ptr[0];
        rows_bytes = form == QUANT_NORM ? 4ull * M * K : head.range[0];
        want = form == QUANT_NORM ? (head.push[6] ? QUANT_F16 : QUANT_PLAIN) : form;
    }
    const LaunchArgs* more[kFuseMax];
    uint32_t n_more = 0;
    uint64_t mask = 0;
    for (uint32_t j = i + 1; j < n && j <= i + kLookahead && n_more + 1u < kFuseMax; ++j) {
        if (ops[j].done) continue;
        const LaunchArgs& q = ops[j].args;
        QuantForm f;
        uint32_t sch;
        if (quant_of(ops[j], &f, &sch) && f != QUANT_NORM && q.ptr[0] == rows_ptr && check_quant(q, f, sch) == AC_SUCCESS) {
            bool ok;
            if (!first) {   // the quantize that says how the gated elements form rows
                ok = (uint64_t)q.push[0] * q.push[1] * 4u == rows_bytes && q.push[2] == q.push[1] && q.push[1] <= 32768u;
            } else {
                const uint32_t stride = form == QUANT_NORM || swiglu ? K : first->push[2];
                ok = f == want && sch == scheme && q.push[0] == M && q.push[1] == K && q.push[2] == stride && q.push[3] == first->push[3];
            }
            ok = ok && can_hoist(ops, i, j, mask);
            // what it writes meets nothing that the head or another member reads or writes
            const uint32_t outs = f == QUANT_F16 ? 5u : 3u;
            for (uint32_t b = 1; b < outs && ok; ++b) {
                ok = !touches(head, q.ptr[b], q.range[b]) && !(first && first != &head && touches(*first, q.ptr[b], q.range[b]));
                for (uint32_t m = 0; m < n_more && ok; ++m) ok = !touches(*more[m], q.ptr[b], q.range[b]);
                for (uint32_t h = 1; h < b && ok; ++h) ok = !overlap(q.ptr[h], q.range[h], q.ptr[b], q.range[b]);
            }
            if (ok) {
                if (first) {
                    more[n_more++] = &q;
                } else {
                    first = &q;
                    form = want = f;
                    scheme = sch;
                    M = q.push[0];
                    K = q.push[1];
                }
                mask |= 1ull << (j - i);
                continue;
            }
        }
        if (!confined(ops[j])) break;
    }
    if (!mask) return AC_SUCCESS;
    *taken = true;
    ops[i].done = true;
    for (uint32_t k = 0; k <= kLookahead; ++k)
        if (mask >> k & 1u) ops[i + k].done = true;
    return launch_quant_group(form, scheme, *first, more, n_more, swiglu ? &head : nullptr);
}

}  // namespace

AcResult launch_fused(FuseOp* ops, uint32_t n, uint32_t i) {
    bool taken = false;
    AcResult rc = AC_SUCCESS;
    QuantForm form;
    uint32_t scheme;
    if (is(ops[i], launch_swiglu_f32) || quant_of(ops[i], &form, &scheme)) {
        rc = fuse_quant(ops, n, i, &taken);
        if (taken) return rc;
    }
    if (is(ops[i], launch_bitnet_norm_q8) || is(ops[i], launch_rms_norm_f32) || is(ops[i], launch_swiglu_f32))
        rc = fuse_bitnet_rows(ops, n, i, &taken);
    else if (is(ops[i], launch_bitnet_gemv_i2_s))
        rc = fuse_bitnet_gemv(ops, n, i, &taken);
    else if (is(ops[i], launch_mmvqb_q6_K) || is(ops[i], launch_mmvqb_q5_K) || is(ops[i], launch_mmvqb_iq4_xs) ||
             is(ops[i], launch_mmvq_q4_1) || is(ops[i], launch_mmvqb_q3_K) || is(ops[i], launch_mmvqb_q2_K))
        rc = fuse_product_add(ops, n, i, &taken);
    else if (is(ops[i], launch_rope) || is(ops[i], launch_set_rows))
        rc = fuse_row_ops(ops, n, i, &taken);
    if (taken) return rc;
    ops[i].done = true;
    return ops[i].entry->launch(ops[i].args);
}

}  // namespace amv
