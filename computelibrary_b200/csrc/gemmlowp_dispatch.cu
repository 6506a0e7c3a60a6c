// Chooses between the builds of the tensor-core kernels (four, eight or sixteen epilogue warps, see
// gemmlowp_tcgen05.cu).  The main loop of a 128 x 256 tile takes about 128 clocks per 32 bytes of K; its
// epilogue takes a fixed few thousand clocks with four warps.  Up to kShortK the epilogue is the longer of the
// two and gets eight warps; beyond it the main loop is, and extra resident warps only slow its single-thread
// producer and MMA loops down.
#include "kernels.cuh"

namespace cugl
{
namespace
{
constexpr int kShortK = 1024;

bool eight_epilogue_warps(const GemmOperands &op)
{
    if (op.epi_warps == 4 || op.epi_warps == 8)
    {
        return op.epi_warps == 8; // forced by the caller (tests, measurements)
    }
    return op.K <= kShortK;
}

// Tile width of the one-CTA kernels.  The widest tile N calls for moves the fewest operand bytes per output, but
// an output of fewer such tiles than SMs leaves SMs idle while each busy one walks all of K for a wide tile.
// Then the width is the one that minimises (waves of tiles over the SMs) x (128 + width), the operand bytes a
// CTA stages per K step; ties go to the wider tile.
int pick_block_n(const cugl_context *ctx, const GemmOperands &op)
{
    const int widest = op.N > 128 ? 256 : (op.N > 64 ? 128 : 64);
    if (op.block_n > 0)
    {
        return op.block_n < widest ? op.block_n : widest;
    }
    if (op.epi_warps == 16 || op.channel_major > 0)
    {
        return widest; // kernels the caller asked for by name: 256-column tiles only
    }
    const long long sms     = ctx->sm_count > 0 ? ctx->sm_count : 1;
    const long long m_tiles = static_cast<long long>((op.M + 127) / 128) * (op.batch > 1 ? op.batch : 1);
    if (m_tiles * ((op.N + widest - 1) / widest) >= sms)
    {
        return widest;
    }
    int       best      = widest;
    long long best_cost = -1;
    for (int bn = widest; bn >= 64; bn >>= 1)
    {
        const long long tiles = m_tiles * ((op.N + bn - 1) / bn);
        const long long cost  = ((tiles + sms - 1) / sms) * (128 + bn);
        if (best_cost < 0 || cost < best_cost)
        {
            best      = bn;
            best_cost = cost;
        }
    }
    return best;
}

// CTAs that share the K range of one 64-column tile.  An output of few tiles leaves SMs idle while each busy one walks all
// of K (about 0.2 us per 128 bytes of K); a cluster of CTAs per tile divides the walk at the price of a cluster launch and
// one exchange of partial sums (1.5 - 2 us).  Measured, back-to-back launches, one CTA / four / eight per tile:
// 49 x 512 x 2048: 8.0 / 7.4 / 6.8 us, 16 x 1024 x 4096: 11.6 / 8.8 / 14.4 (eight: more CTAs than SMs), 256 x 1024 x 4096
// to float32 11.8 / 9.0, 64 x 1024 x 1024: 6.0 / 6.7; 3x3 convolutions, whose patch loads take longer, 1 x 7 x 7 x 512:
// 18.1 / 10.7 / 8.5, 1 x 14 x 14 x 256: 11.1 / 8.8 / 7.8, 1 x 28 x 28 x 128 (K = 1152): 8.1 / 7.7 / 7.7.  Two per tile gain
// nothing (16 x 4096 x 4096: 11.7 / 11.9).  Eight-CTA clusters need their SMs inside one GPC, hence the margins.
int pick_split(const cugl_context *ctx, const GemmOperands &op)
{
    if (op.batch > 1 || op.n_extra_dst > 0 || op.channel_major > 0 || op.block_n > 0 || op.epi_warps != 0 ||
        (op.conv != nullptr && op.conv->C == 64))
    {
        return 1;
    }
    const long long tiles = static_cast<long long>((op.M + 127) / 128) * ((op.N + 63) / 64);
    const int       kb    = (op.K + 127) / 128;
    if (kb >= 16 && tiles * 8 <= ctx->sm_count * 3 / 4) return 8;
    if (kb >= (op.conv != nullptr ? 9 : 16) && tiles * 4 <= ctx->sm_count * 9 / 10) return 4;
    return 1;
}

// 8-bit rows of dst that are not 16-byte aligned cannot leave as bulk tensor stores.  The channel-major kernel with sixteen
// warps, whose lanes write eight neighbouring rows' bytes of their channel, is the fastest way out for them wherever its
// 128-channel x 256-row tiles occupy half the device; against the row-major kernel's staged words (eight warps), us:
// 2099 x 3709 x 352 13.5 / 20.7, 4000 x 5001 x 64 26.8 / 45.3, x 1000 39.7 / 54.7, 8000 x 301 x 256 8.4 / 11.8,
// 500 x 6001 x 352 8.8 / 12.1, and with a single block of channels 100000 x 65 x 256 17.7 / 24.6, 20000 x 65 x 64 7.9 / 10.6; up
// to 64 channels half of the tile and more is empty (100000 x 63 x 256 17.5 / 16.9, x 33 18.1 / 16.5, x 17 18.1 / 13.4).  The
// bound on K is where the row-major kernels change, not a crossing: 2099 x 3709 x 2000 25 / 34.
bool ragged_rows_channel_major(const cugl_context *ctx, const GemmOperands &op)
{
    const bool      aligned = ((reinterpret_cast<uintptr_t>(op.dst) | static_cast<uint64_t>(op.ldd)) & 15) == 0;
    const long long tiles   = static_cast<long long>((op.N + 127) / 128) * ((op.M + 255) / 256);
    return !aligned && op.channel_major == 0 && op.epi_warps == 0 && op.block_n == 0 && op.batch <= 1 && op.n_extra_dst == 0 &&
           op.conv == nullptr && op.N > 64 && op.K <= kShortK && tiles >= ctx->sm_count / 2;
}

// Four or eight epilogue warps for a batch in one launch.  The batched kernels fill every wave, so that the shorter main
// loop of four warps pays later than in single products, us with eight / four: 2 x 2432 x 2432 x 1152 18.9 / 19.6,
// 4 x 1500^3 (ragged rows) 32 / 38, 2 x 8192 x 2048 x 1280 40.8 / 39.1, 4 x 2304 x 2304 x 1536 36.7 / 32.8,
// 2 x 2048 x 2304 x 8192 to float32 77 / 69.  Ragged 8-bit rows leave through the staged words, which want eight warps until
// the main loop hides them: 2 x 4000 x 5001 x 2000 99 / 127, 2 x 2500 x 2501 x 4096 55.9 / 54.8.
bool batch_eight_epilogue_warps(const GemmOperands &op, bool output_stage)
{
    if (op.epi_warps == 4 || op.epi_warps == 8)
    {
        return op.epi_warps == 8;
    }
    const bool ragged = output_stage && ((reinterpret_cast<uintptr_t>(op.dst) | static_cast<uint64_t>(op.ldd)) & 15) != 0;
    return op.K < (ragged ? 4096 : 1280);
}

// the SM-pair kernel works on 256 x 256 tiles, one per pair of SMs
bool pair_fills_the_device(const cugl_context *ctx, const GemmOperands &op)
{
    const long long tiles = static_cast<long long>((op.M + 255) / 256) * ((op.N + 255) / 256);
    return tiles >= ctx->sm_count / 2;
}
} // namespace

bool gemmlowp_conv_tma_supported(const GemmOperands &op)
{
    return gemmlowp_conv_tma_supported_epi4(op);
}

bool gemmlowp_tcgen05_supported(const GemmOperands &op)
{
    return gemmlowp_tcgen05_supported_epi4(op);
}

// The SM-pair kernel pays off once a tile spans both halves (more than 128 rows and more than 128 columns), the
// main loop is long enough to matter and there is a 256 x 256 tile for every pair of SMs.
bool gemmlowp_tcgen05_uses_pair(const cugl_context *ctx, const GemmOperands &op)
{
    return gemmlowp_tcgen05_uses_pair_epi4(op) && !eight_epilogue_warps(op) && pair_fills_the_device(ctx, op) &&
           (op.block_n == 0 || op.block_n == 256);
}

// The batched launch runs the one-CTA row-major kernels.  What its products lose by that, one by one / in one launch, us:
// * the SM-pair kernel, where K is long and one product's 256 x 256 tiles come in nearly whole waves of SM pairs:
//   4 x 4096^3 199 / 207, 3 x 4096 x 2048 x 4096 86 / 90; not 4 x 3072^3 (99 / 96), nor 2 x 4096 x 4096 x 2048 (56.1 / 57.4, to
//   float32 69.8 / 69.2), nor 2 x 2560 x 2560 x 2048 (1.4 waves: 33 / 27);
// * the channel-major kernel for ragged 8-bit rows: 2 x 2099 x 3709 x 352 26.9 / 39.0, 3 x 4000 x 5001 x 256 80 / 119,
//   2 x 1200 x 2001 x 400 18.4 / 21.4, 2 x 8000 x 1001 x 1000 46 / 51; not where one product's tiles are little more than
//   a wave (4 x 1000 x 5001 x 256, 160 tiles: 50.1 / 46.7), nor a part of one above K = 512 (2 x 1200 x 3001 x 900: 29.7 / 27.8).
// Everything else gains: 8 x 1024^3 50 / 13.3, 4 x 4096 x 4096 x 1024 103 / 65, 2 x 50176 x 256 x 64 24.8 / 18.8.
bool gemmlowp_batch_by_product(const cugl_context *ctx, const GemmOperands &op, bool output_stage, bool allow_pair)
{
    auto whole_waves = [](long long tiles, long long slots) { return 5 * tiles >= 4 * slots * ((tiles + slots - 1) / slots); };
    const long long sms = ctx->sm_count;
    const long long pair_tiles = static_cast<long long>((op.M + 255) / 256) * ((op.N + 255) / 256);
    if (allow_pair && op.K >= 4096 && gemmlowp_tcgen05_uses_pair(ctx, op) && whole_waves(pair_tiles, sms / 2))
    {
        return true;
    }
    const long long cm_tiles = static_cast<long long>((op.N + 127) / 128) * ((op.M + 255) / 256);
    return output_stage && ragged_rows_channel_major(ctx, op) && (cm_tiles > sms ? whole_waves(cm_tiles, sms) : op.K <= 512);
}

cugl_status launch_gemmlowp_tcgen05(cugl_context *ctx, const GemmOperands &op, const EpilogueParams &ep,
                                    bool allow_pair)
{
    // The channel-major kernel (operand roles exchanged, output-stage terms in registers, stores through a byte
    // transpose in shared memory) against the row-major one with sixteen epilogue warps, paired drain and 256-bit
    // stores, measured: 802816 x 256 x 64: 189 us against 170 us; 200704 x 512 x 128: 102 / 94; 50176 x 1024 x 256:
    // 57 / 60; 12544 x 2048 x 512: 37 / 43.  It needs whole 128-channel blocks (N = 64: 110 / 78).
    GemmOperands o   = op;
    const int split = pick_split(ctx, op);
    if (split > 1)
    {
        o.split_k       = split;
        o.channel_major = -1;
        return launch_gemmlowp_tcgen05_epi8(ctx, o, ep, false);
    }
    if (ep.stage != CUGL_STAGE_NONE && ep.rowsum == nullptr && ragged_rows_channel_major(ctx, op))
    {
        o.channel_major = 1;
        return launch_gemmlowp_tcgen05_epi16(ctx, o, ep, false);
    }
    o.block_n        = pick_block_n(ctx, op); // before the automatic channel-major choice below
    if (op.batch > 1)
    {
        // Batches of attention-sized products: their tiles share one grid instead of each product filling its own
        // (16 products of 384 x 384 x 128: 6 - 18 tiles each).
        return batch_eight_epilogue_warps(o, ep.stage != CUGL_STAGE_NONE) ? launch_gemmlowp_tcgen05_epi8(ctx, o, ep, false)
                                                                          : launch_gemmlowp_tcgen05_epi4(ctx, o, ep, false);
    }
    if (ep.stage == CUGL_STAGE_NONE && (ep.out_f32 != 0 || ep.accumulate != 0) && o.channel_major == 0)
    {
        o.channel_major = -1; // read-modify-write of dst rows: the row-major epilogue does it row by row, 128 bytes at a time
    }
    if (o.channel_major == 0)
    {
        // with a fused residual too: 50176 x 1024 x 256 + residual 69 us against 79 us row-major, 12544 x 2048 x 512
        // 43 / 53; below K = 256 the two are level with a residual (200704 x 512 x 128: 125 / 128) and the row-major
        // kernel is ahead without one (102 / 94)
        // since the row-major epilogue stores through the TMA unit the two were measured again (batch 256, row-major /
        // channel-major): 256 -> 1024 at 14 x 14 45 / 45 us (with a residual 64 / 60), 256 -> 512 at 28 x 28 74 / 84,
        // 1024 -> 256 27 / 29, 512 -> 1024 53 / 49, 512 -> 2048 at 7 x 7 37 / 31, 1024 -> 2048 41 / 37
        o.channel_major = (o.K >= 512 && o.K <= kShortK && o.N >= 1024) ? 1 : -1;
    }
    const int widest = o.N > 128 ? 256 : (o.N > 64 ? 128 : 64);
    if (o.block_n < widest)
    {
        // a small output: narrower tiles on more SMs (the kernels of the complete builds only)
        o.channel_major = -1;
        return eight_epilogue_warps(o) ? launch_gemmlowp_tcgen05_epi8(ctx, o, ep, false)
                                       : launch_gemmlowp_tcgen05_epi4(ctx, o, ep, false);
    }
    allow_pair = allow_pair && pair_fills_the_device(ctx, o);
    // sixteen epilogue warps (256-column tiles only) buy another 4 - 7 % on short K with wide outputs
    // (up to K = 512, where its paired drain applies; above, eight warps -- whose single-tile drain stores through the
    // TMA unit -- measured faster: 50176 x 256 x 1024 25.5 against 27.6 us)
    // Rows of dst that are not 16-byte aligned: only the smaller builds stage those, the sixteen-warp row-major drain writes
    // them byte by byte (2099 x 3709 x 352: 91 us against 21 with eight warps, 8000 x 1001 x 64: 87 / 20); channel-major
    // keeps its sixteen (4000 x 5001 x 512: 28 / 37).
    const bool dst_rows = ((reinterpret_cast<uintptr_t>(o.dst) | static_cast<uint64_t>(o.ldd)) & 15) == 0;
    if (o.N > 128 && (o.epi_warps == 16 || ((dst_rows || o.channel_major > 0) && ep.stage != CUGL_STAGE_NONE && o.epi_warps != 4 && o.epi_warps != 8 && o.K <= 512)))
    {
        return launch_gemmlowp_tcgen05_epi16(ctx, o, ep, false);
    }
    return eight_epilogue_warps(o) ? launch_gemmlowp_tcgen05_epi8(ctx, o, ep, false)
                                   : launch_gemmlowp_tcgen05_epi4(ctx, o, ep, allow_pair);
}

bool gemmlowp_conv_tcgen05_supported(const GemmOperands &op, const ConvOperands &cv)
{
    return gemmlowp_conv_tcgen05_supported_epi4(op, cv);
}

cugl_status launch_gemmlowp_conv_tcgen05(cugl_context *ctx, const GemmOperands &op, const EpilogueParams &ep,
                                         const ConvOperands &cv)
{
    GemmOperands o = op;
    o.block_n      = pick_block_n(ctx, o);
    return eight_epilogue_warps(o) ? launch_gemmlowp_conv_tcgen05_epi8(ctx, o, ep, cv)
                                   : launch_gemmlowp_conv_tcgen05_epi4(ctx, o, ep, cv);
}
} // namespace cugl
