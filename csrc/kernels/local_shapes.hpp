/**
 * Which shape the one-GPU copy and the pairwise fold (local.cu) run in, by size. Both sides of each line were timed in turn on one
 * B200 with "one" pair of buffers again and again, "three" pairs in turn, and as many pairs as it takes to find nothing of a pair
 * in L2 (126 MB) again, "HBM". Times are microseconds per call, given in this order.
 */
#pragma once
#include <cstddef>

namespace dccl {

/**
 * Threads of a CTA of the copy. CTAs of 1024 stream 1 to 2 % faster out of HBM, CTAs of 256 are up to 17 % faster out of L2; the line
 * lies where L2 keeps nothing of a pair. 256 -> 1024 threads: 28 MiB 5.72 -> 6.22, 10.14 -> 9.99, 10.24 -> 10.11; 64 MiB 18.28 ->
 * 19.53, 21.04 -> 20.86, 21.19 -> 20.91; 72 MiB 22.86 -> 22.91, 23.53 -> 23.17, 23.60 -> 23.19; 80 MiB 25.85 -> 25.50, 26.01 ->
 * 25.60, 26.04 -> 25.68; 1 GiB 309 -> 305 in all three. From a source 6 bytes off: 64 MiB 19.07 -> 20.57, 21.15 -> 21.09, 21.25 ->
 * 21.02; 80 MiB 25.91 -> 25.98, 26.09 -> 25.86, 26.04 -> 25.88; 100 MiB 32.18 -> 31.77, 32.07 -> 31.95, 32.05 -> 31.90.
 */
constexpr unsigned copy_threads(size_t bytes) { return bytes >= (80u << 20) ? 1024 : 256; }

/**
 * Whether a thread of the fold takes two vectors, in CTAs of 128, or one, in CTAs of 512; bytes of one operand. Two are ahead out of
 * L2, one out of HBM, and the band is where two gain for one pair and for three alike: 1 to 9 % and 3 to 14 % in fp32, fp64, bf16,
 * bytes, products and operands at odd elements. Operands out of HBM take up to 2.2 % longer there (bf16 0.8 % on average). A
 * single pair would gain from 6 to 64 MiB, by 18 % at 56, which three pairs in turn pay for with 2 to 4 % at 8 and 1 % from 28 MiB
 * on. bf16 sum, one -> two vectors: 8 MiB 2.77 -> 2.75, 2.77 -> 2.77, 5.29 -> 5.33; 10 MiB 3.36 -> 3.19, 3.35 -> 3.19, 6.16 -> 6.20;
 * 16 MiB 4.50 -> 4.38, 7.13 -> 6.22, 8.83 -> 8.90; 22 MiB 5.67 -> 5.43, 11.21 -> 10.58, 11.47 -> 11.56; 25 MiB 6.28 -> 6.01, 12.78
 * -> 12.67, 12.84 -> 12.91; 28 MiB 6.86 -> 6.48, 13.94 -> 14.05, 14.05 -> 14.20; 56 MiB 24.75 -> 20.30, 26.19 -> 26.50, 26.29 ->
 * 26.70; 256 MiB 113 -> 115 in all three.
 */
constexpr bool two_vectors(size_t bytes) { return bytes >= (10u << 20) && bytes <= (22u << 20); }

} // namespace dccl
