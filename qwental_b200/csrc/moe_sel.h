// Selection record shared by the MoE kernels and the fused combine + norm kernel.
#pragma once
#include <stdint.h>

#define MOE_MAXB 64
#define MOE_MAXK 16
#define MOE_MAXE 1024

// Result of the selection, read by the gate/up, down and combine kernels (role of struct gg_sel,
// kernels/moe_gg.metal:110-116).  Groups are in expert-id order; a group's entries are in token order.
// MAXB = 64: a step.  MAXB = 1024: a piece of a prompt; the fields up to w sit at the same offsets in both.
template <int MAXB>
struct moe_sel_t {
    uint32_t U;                               // groups (distinct experts in [e_lo, e_hi) that were chosen)
    uint32_t nb, topk, pad;
    int32_t ids[MOE_MAXB][MOE_MAXK];          // chosen experts of the first 64 tokens, rank order
    float w[MAXB][MOE_MAXK + 1];              // routed weights, then the shared gate at [topk]
    uint32_t ue[MOE_MAXE];                    // expert of group u
    uint32_t off[MOE_MAXE + 1];               // entries of group u: ent[off[u] .. off[u+1])
    static constexpr int TOK = MAXB > 256 ? 4 : 8;  // bits of an entry below its token
    uint16_t ent[MAXB * MOE_MAXK];            // token << TOK | rank
    uint32_t pre[MOE_MAXE + 2];               // passes of 8 entries in the groups before u (pre[U] = all routed passes)
};
typedef moe_sel_t<MOE_MAXB> moe_sel;
#define MOE_MAXB_WIDE 1024
struct moe_sel_wide : moe_sel_t<MOE_MAXB_WIDE> {
    uint16_t sid[MOE_MAXB_WIDE][MOE_MAXK];    // chosen experts of every token: from the top-k to the grouping
    uint32_t prw[MOE_MAXE + 2];               // items of the expert FFN (MOE_FFN_COLS_WIDE entries each) in the groups before u
};

// Scratch buffer of the fused expert-FFN kernel (k_ffn.cu): the items' counters and the finished-block counter in the first
// MOE_FFN_SYNC_BYTES (all zero between launches: the owner zeroes the buffer once), then H [item][2 planes][8 columns][I] fp16.
// An item is one pass of up to 8 tokens of one chosen expert or of the shared expert: at most 512 experts + the extra passes
// of 64 tokens x 10 choices + the shared expert's 8.
#define MOE_FFN_MAXITEMS 640
#define MOE_FFN_SYNC_BYTES 8192
// word MOE_FFN_ROWCNT + tok * (topk + 1) + rank of the same area counts the reader warps that have stored their part of output row
// (tok, rank) of Pg: 8 per tile of 128 output rows, MOE_FFN_ROW_DONE(D) when the row is complete.  The combine + norm kernel that
// follows waits on the rows of its token instead of on the whole launch, and clears them (one GPU only).
#define MOE_FFN_ROWCNT 1024
#define MOE_FFN_ROW_DONE(D) ((D) / 128 * 8)
#define MOE_FFN_SCRATCH_BYTES(I) ((size_t)MOE_FFN_SYNC_BYTES + (size_t)MOE_FFN_MAXITEMS * 16 * (I) * 2)
// The same for a piece of a prompt of up to ROWS tokens, in a buffer of its own.  An item has up to MOE_FFN_COLS_WIDE columns.  H is [entry, then the
// shared expert's tokens][2 planes][I].  No output row is counted in.
#define MOE_FFN_COLS_WIDE 16
#define MOE_FFN_MAXITEMS_WIDE (512 + MOE_MAXB_WIDE * MOE_MAXK / MOE_FFN_COLS_WIDE)
#define MOE_FFN_SYNC_BYTES_WIDE 8192
#define MOE_FFN_SCRATCH_BYTES_WIDE(I, ROWS) ((size_t)MOE_FFN_SYNC_BYTES_WIDE + (size_t)(ROWS) * MOE_MAXK * 2 * (I) * 2)
