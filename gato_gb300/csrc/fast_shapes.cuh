// Shapes of the register-resident two-pass engine: M = 2N -> (R1, R2, lines per CTA FP32, FP64, FP32
// strands accumulating, to J).
// R1 and R2 are even: the zero-padded half of every transform maps to whole register slots, and the
// x pass folds the kernel spectrum at R2 / 2. Every even N from 16 to 144 whose 2N factors into 2, 3, 5
// and 7 has one (and N = 160); the rest, smaller and odd N among them, takes the Stockham engine. On FP32 fields that
// engine is 1.6 (N = 18) to 6 (N = 144) times slower than these shapes (exchange with four orbitals:
// 462 against 167 us at N = 100, 2088 against 347 at 144); on FP64 fields, where the FP64 pipe binds
// both, 0 to 25 % (1146 against 917 us at N = 72).
// Lines per CTA: 16 puts every stage of an even radix on whole warps, which an FP64 stage needs (a
// half-empty warp costs the narrow pipe a whole one) even where the last tile of columns is then partly
// idle; the others are those of a sweep over 8 to 32 lines that beat it, by 1 to 6 % of the column
// passes (FP64: M = 200 2802 us at 16 lines, 2661 at 8; FP32: M = 280 269 and 248).
// FP32 strands: the most fields that two strands transform faster than one, accumulating and to J fields (0: never,
// 40: any number; two_strands in poisson.cu has the figures). FP64 fields always gain.
// Groups are translation units of similar size.
#pragma once

#define GATO_FAST_SHAPES_0(X) \
  X(32, 4, 8, 32, 16, 0, 0) X(48, 6, 8, 32, 16, 0, 0) X(64, 8, 8, 32, 16, 0, 0) \
  X(80, 10, 8, 32, 16, 0, 0) X(96, 8, 12, 16, 8, 0, 0) X(128, 8, 16, 16, 8, 40, 40) \
  X(36, 6, 6, 16, 16, 0, 0) X(40, 10, 4, 16, 8, 0, 0)
#define GATO_FAST_SHAPES_1(X) \
  X(160, 10, 16, 16, 16, 40, 40) X(192, 12, 16, 16, 8, 40, 40) X(256, 16, 16, 16, 8, 40, 40) \
  X(320, 20, 16, 16, 8, 40, 40)
#define GATO_FAST_SHAPES_2(X) \
  X(56, 14, 4, 16, 8, 0, 0) X(60, 10, 6, 16, 12, 0, 0) X(72, 12, 6, 16, 16, 0, 0) \
  X(84, 14, 6, 16, 14, 0, 0) X(100, 10, 10, 16, 16, 0, 0) X(108, 18, 6, 16, 16, 0, 0) \
  X(112, 14, 8, 16, 16, 0, 0) X(120, 12, 10, 16, 8, 0, 0) X(140, 14, 10, 16, 16, 5, 5)
#define GATO_FAST_SHAPES_3(X) \
  X(144, 12, 12, 16, 8, 5, 5) X(168, 14, 12, 16, 16, 5, 3) X(180, 18, 10, 16, 12, 4, 3) \
  X(196, 14, 14, 16, 16, 2, 2) X(200, 20, 10, 16, 8, 5, 5) X(216, 18, 12, 16, 16, 2, 2) \
  X(224, 14, 16, 16, 16, 2, 5) X(240, 20, 12, 16, 8, 5, 2) X(252, 18, 14, 16, 16, 2, 2) \
  X(280, 20, 14, 8, 8, 2, 2) X(288, 18, 16, 16, 16, 0, 2)
#define GATO_FAST_SHAPES_ALL(X) \
  GATO_FAST_SHAPES_0(X) GATO_FAST_SHAPES_1(X) GATO_FAST_SHAPES_2(X) GATO_FAST_SHAPES_3(X)
