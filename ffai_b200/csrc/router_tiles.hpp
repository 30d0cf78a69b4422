// Which tiles the router projection of a long prompt takes: 128 tokens x 64 experts (two blocks per SM) or 128 x 128 (one).
#pragma once

namespace ffai {

// `tiles`: narrow tiles of the batch; the experts make an even count of narrow columns (a last column of at most 64 experts
// would leave half a wide tile empty).  A round of wide tiles over the SMs takes as long as almost two of narrow ones, so the
// wide tiles pay where the narrow ones need an even count of rounds, and lose most of a round where it is odd.  us, H = 2048,
// wide / narrow:
//   narrow rounds     2 (8192 x 256)   3 (12288)     4 (16384)     5 (21504)     6 (24576)     7 (32768)
//   bf16 weights      236 / 274        449 / 410     457 / 524     673 / 659     680 / 773     896 / 915
//   fp32 weights      256 / 270        491 / 399     499 / 522     731 / 650     737 / 768     977 / 913
// One round: the narrow tiles, with the hidden axis split (64 tiles 87 us).
constexpr bool router_wide_tiles(int tiles, int n_sms, bool fp32) {
    const int rounds = (tiles + n_sms - 1) / n_sms;
    return rounds > 1 && (rounds % 2 == 0 || (!fp32 && rounds >= 7));
}

}  // namespace ffai
