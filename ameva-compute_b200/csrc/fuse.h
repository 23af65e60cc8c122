// Recorded dispatches that leave the host in one launch. A batch is launched in the order it was recorded; where a run of
// its dispatches has a fused form, fuse.cu launches that form instead, with the same results in the same buffers (every
// destination a separate dispatch would have written is written). At token generation a layer is a chain of launches of 2-4
// us whose work takes a fraction of that, so the number of launches is what it costs.
#pragma once
#include "common.cuh"

namespace amv {

struct FuseOp {
    const KernelEntry* entry;
    LaunchArgs args;
    bool done;   // launched, alone or as part of a fused form
    enum { UNKNOWN, PASSES, REFUSED } checks;   // of its launcher, where a later operation is to run before it
};

// Launches ops[i] together with the later operations that can join it, and marks all of them done.
AcResult launch_fused(FuseOp* ops, uint32_t n, uint32_t i);

// ---- fused forms (each launcher validates what the separate launchers validate; the matching is in fuse.cu) ------------
constexpr uint32_t kFuseMax = 4;   // members of a group

// bitnet rows (act_quant.cu): the quantize of an I2_S product over rows that are copied (PLAIN), RMS-normalised (NORM, the
// arguments of ameva_rms_norm_f32) or formed by SWIGLU (ameva_swiglu_f32) by the dispatch before, written to n destinations
enum BitnetSource { BITNET_PLAIN, BITNET_NORM, BITNET_SWIGLU };
AcResult check_bitnet_norm_q8(const LaunchArgs& a);
bool bitnet_rows_fits(const LaunchArgs& norm_q8);   // a plain quantize (mode 0, no norm) the row kernel serves
AcResult launch_bitnet_rows(BitnetSource source, const LaunchArgs* head, const LaunchArgs* const* norm_q8, uint32_t n);

// up to four I2_S products (bitnet_gemv_i2_s_*) of the same K and row count (1 or 2) in one launch; add: with n == 1, the
// ameva_add_f32 whose first (swapped: second) operand is the product
AcResult check_bitnet_gemv_i2_s(const LaunchArgs& a);
AcResult launch_bitnet_gemv_i2_s_group(const LaunchArgs* const* gemv, uint32_t n, const LaunchArgs* add, bool swapped);

// the quantize kernels (act_quant.cu), per-32 (scheme 0) and per-256 (scheme 1): several that read the same rows (the first
// may be the fused RMS norm + quantize that writes them) in one pass, or the SWIGLU that forms the rows with them
enum QuantForm { QUANT_PLAIN, QUANT_F16, QUANT_NORM };
AcResult check_quant(const LaunchArgs& a, QuantForm form, uint32_t scheme);
AcResult launch_quant_group(QuantForm form, uint32_t scheme, const LaunchArgs& first, const LaunchArgs* const* more, uint32_t n_more,
                            const LaunchArgs* swiglu);

// ROPE / SET_ROWS of the same new positions (layer_ops.cu): up to two of each beside one another, and per ROPE a SET_ROWS of
// its result (store[i], nullptr: none)
bool row_op_serves(const LaunchArgs& a, bool rope);
bool rope_feeds_set_rows(const LaunchArgs& rope, const LaunchArgs& set);
AcResult launch_row_ops(LaunchStream stream, const LaunchArgs* const* rope, const LaunchArgs* const* store, uint32_t n_rope,
                        const LaunchArgs* const* set, uint32_t n_set);

}  // namespace amv
