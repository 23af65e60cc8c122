// Arguments of ameva_flash_attn (the reference's 31 push words, ameva_flash_attn.comp:46-58) and the interface between its
// launcher (layer_ops.cu) and the tensor-core kernel for prompts (flash_tc.cu).
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace amv {

struct LaunchArgs;

struct FlashArgs {
    uint32_t D, DV, n_kv, n_q;
    uint32_t n_head, n_head_kv, kv_types, has_mask;
    uint32_t q_off, q_s1, q_s2, k_off;
    uint32_t k_s1, k_s2, v_off, v_s1;
    uint32_t v_s2, m_off, m_s1, m_s2;
    uint32_t m_ne2, o_off, scale, softcap;
    uint32_t max_bias, m0, m1, n_head_log2;
    uint32_t tile_base;
    uint32_t split_keys, part_off;
};

struct FlashMaps {
    CUtensorMap k, v;
};

constexpr uint32_t kFlashTcRows = 128, kFlashTcKeys = 64, kFlashTcPerSm = 2;   // rows per CTA, keys per tile, CTAs per SM

// The tensor maps of K and V; false where the strides cannot be expressed in one.
bool flash_tc_maps(const LaunchArgs& a, const FlashArgs& pc, FlashMaps* maps);
// split_keys: a multiple of kFlashTcKeys; q_tiles = ceil(n_q / (kFlashTcRows / G)).
bool launch_flash_tc(const LaunchArgs& a, const FlashMaps& maps, const FlashArgs& pc, uint32_t n_splits, uint32_t q_tiles);

}  // namespace amv
