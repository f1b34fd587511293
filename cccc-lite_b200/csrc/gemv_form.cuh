// Which form of the decode kernel a linear of up to 8 tokens takes, and how its k range is dealt out.  Host code without CUDA, so that
// the rules can be looked at without a GPU.
#pragma once

#include <cstddef>

namespace b200
{

enum class GemvForm
{
    Low,     // row blocks of 32 rows, eight warps; stages of 2048 k at 1 and 2 tokens, of 1024 (FP4: twice as many) above
    Long,    // 3 to 8 tokens: the same with stages of 2048 k
    Tall     // row blocks of 64 rows, sixteen warps, stages of 1024 k
};

// Are whole row blocks dealt out, so that nothing is exchanged between CTAs, or is the k range split as well (stream-K)?
// Measured on B200: the exchange costs about 5 us of serial latency, one SM alone streams about 45 GB/s; so the k range is only split
// when whole row blocks would leave most SMs idle for long.
static inline bool gemv_whole_blocks(unsigned int block_rows, bool fp4, unsigned long long row_blocks, unsigned int K, int sm_count)
{
    const double block_bytes = (double)block_rows * (double)(fp4 ? K / 2 + K / 16 : K), sms = (double)sm_count;
    const double rounds = (double)((row_blocks + (unsigned)sm_count - 1) / (unsigned)sm_count);
    const double t_whole = rounds * block_bytes / 45e9;
    const double t_split = 5e-6 + (double)row_blocks * block_bytes / (sms * 40e9);
    return t_whole <= t_split;
}

// Row blocks of 64 rows and sixteen warps, or of 32 and eight (low, tall: the launch's row blocks of either height)?  Twice the warps keep a stage's
// conversions going better (at 1 token, 32 / 64 rows, us: E4M3 6144 x 4096 10.1 / 8.9, 24576 x 4096 26.2 / 24.5, 151936 x 4096 120.1 / 113.8; E5M2 9.0 /
// 7.8, 22.5 / 21.3, 101.3 / 95.4), but whole blocks are dealt out: it is for launches whose busiest SM then has no more rows, or hardly more (28672 x
// 4096, 256 rows against 224, 29.0 / 30.9; 4096 x 4096 6.0 / 7.6).  FP8 at 3 to 8 tokens, in stages of 96 KB, gains where every block has an SM of its
// own (6144 x 4096 9.7 / 8.8) and not beyond (151936 x 4096 118.0 / 118.9).  FP4 gains alone (6144 x 4096 at 1 token 9.7 / 8.5) and loses in a layer (8
// tokens, four calls, 49.3 / 50.9: fewer, longer CTAs keep the next kernel's out).
// FP8 of 3 to 8 tokens that stays low: two stages of 96 KB instead of four of 48 where k is whole stages of 2048 (E4M3 at 3 tokens, 48 / 96 KB: 4096 x
// 4096 6.8 / 6.3, 4096 x 12288 14.8 / 13.2, 24576 x 4096 28.4 / 25.3, 151936 x 4096 138.6 / 118.0); FP4, twice the elements per byte, has no room for two such.
//
// A warp's k steps and the order of the sums are the same in all forms as long as whole row blocks are dealt out: so are the bits.  A split
// k range is cut between stages, so the bits follow the form there: such a launch stays low, and so has the bits of the calls that never
// leave that form, the allocation-free ones (partial_bytes is too small) and those with the exchange fused in (world > 1).
static inline GemvForm gemv_form(bool fp4, unsigned int M, unsigned int K, unsigned long long low, unsigned long long tall, int sm_count, int world,
    size_t partial_bytes)
{
    if (fp4 || M > 8 || world > 1 || !gemv_whole_blocks(32, false, low, K, sm_count)) { return GemvForm::Low; }
    const unsigned long long sms = (unsigned long long)sm_count;
    const unsigned long long rows_low = (low + sms - 1) / sms * 32, rows_tall = (tall + sms - 1) / sms * 64;
    const bool even = M > 2 ? rows_tall <= rows_low && tall <= sms : rows_tall * 93 <= rows_low * 100;
    if (even && gemv_whole_blocks(64, false, tall, K, sm_count) && (size_t)sm_count * 2 * 64 * 8 * sizeof(float) <= partial_bytes) { return GemvForm::Tall; }
    return M > 2 && K % 2048 == 0 ? GemvForm::Long : GemvForm::Low;
}

}    // namespace b200
