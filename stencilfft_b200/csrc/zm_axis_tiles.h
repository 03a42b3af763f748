// zm_axis_tiles.h -- the tile shapes compiled for the axis pass sized by N alone
// (zm_axis.cuh): X(log2 N, log2 lines per tile, log2 points per thread, log2 largest digit),
// per N the wide tile first and, where one is listed, the narrow one that fields of few
// lines take.  Measured on B200, forward / inverse microseconds per transform.
//
// Points per thread: 16 complex64 are 32 registers of data, 64 in all, 1024 threads per SM;
// 32 complex64 or 16 complex128 are 64 of 128, 512 threads.  32 points either allow 32-point
// digits, which save a stage (N = 1024 c64 2D 12.1 / 11.6 -> 11.2 / 11.0; 3D N = 512
// 1.43 / 1.43 -> 1.22 / 1.39 ms; N = 8192 1.08 / 0.88 -> 0.73 / 0.76 ms with a second line),
// or give a thread both lines of a tile, which then share the loads of the twiddles (N = 4096
// c64 162 / 166 -> 145 / 169).  N = 8192 complex128 holds 32 points in 255 registers: three
// stages instead of four (1.58 / 1.72 -> 1.42 / 1.59 ms).
// Lines per tile: the strided sides move runs of TL x TL elements (2D) or TL (3D), so 3D
// tiles want 128-byte runs (N = 256 c64 248 / 227 with two lines, 157 / 162 with sixteen).
// More lines than that leave an SM one or two tiles, with little to overlap (N = 4096 c64 2D
// 145 / 169 with two lines, 188 / 195 with four; one line writes half sectors: 241 / 210).
// Narrow tiles: a 2D field of N = 256 has 256 lines, 16 wide tiles for 148 SMs; tiles of four
// lines take 4.9 / 5.1 us against 8.1 / 8.2.
#pragma once

#define ZM_AXIS_TILES_C64(X)           \
    X(4, 3, 4, 4)                      \
    X(5, 3, 3, 3)                      \
    X(6, 3, 3, 3)                      \
    X(7, 4, 4, 4) X(7, 2, 3, 3)        \
    X(8, 4, 4, 4) X(8, 2, 3, 3)        \
    X(9, 4, 5, 5) X(9, 2, 3, 3)        \
    X(10, 2, 5, 5)                     \
    X(11, 1, 5, 4)                     \
    X(12, 1, 5, 4)                     \
    X(13, 1, 5, 5)                     \
    X(14, 0, 5, 5)
#define ZM_AXIS_TILES_C128(X)          \
    X(4, 2, 4, 4)                      \
    X(5, 2, 3, 3)                      \
    X(6, 2, 3, 3)                      \
    X(7, 4, 4, 4) X(7, 2, 3, 3)        \
    X(8, 3, 4, 4) X(8, 1, 4, 4)        \
    X(9, 3, 4, 4) X(9, 2, 4, 4)        \
    X(10, 1, 4, 4)                     \
    X(11, 1, 4, 4)                     \
    X(12, 0, 4, 4)                     \
    X(13, 0, 5, 5)
