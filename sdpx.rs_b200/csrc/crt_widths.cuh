// Register widths of the FP64 form's CRT (k_rns_crt_f64): it keeps two 64-bit accumulators a word in
// registers, so a width too far above the words needed costs instructions on words of zeros and, at 64
// words, more registers than a thread has.  Products of inner size 16 with 16 and 64 words alone and with these
// widths, us: 1000 x 1000 outputs at 64 bits (5 words) 271 and 239, at 128 bits 420 and 383, at 512 bits (20
// words) 4727 and 2570, at 768 bits (500 x 500) 3106 and 2131.
#pragma once

namespace sdpxg {

constexpr int kCrtMaxWords = 64;  // 64-bit words of the reconstructed integer

// The instantiated width for `words` words.
constexpr int crt_f64_words(int words) { return words <= 8 ? 8 : words <= 16 ? 16 : words <= 32 ? 32 : kCrtMaxWords; }

}  // namespace sdpxg
