// Generated by symmetrix-xl_b200/csrc/gen_structures.py -- do not edit.
// Coupling structure of the supported model shapes as X-macro lists.
#pragma once

// ---- shape S0: edge l_max=3, hidden L_max=0
#define SXB_S0_LMAX 3
#define SXB_S0_HIDDEN_LMAX 0
#define SXB_S0_NUM_LM 16
#define SXB_S0_NUM_HIDDEN 1
#define SXB_S0_NUM_PATHS 4
#define SXB_S0_NUM_ROWS 16
#define SXB_S0_NUM_LME 16
#define SXB_S0_NUM_TERMS 16
// X(path, l_out, l_edge, l_source, first_row)
#define SXB_S0_PATHS(X) \
    X(0, 0, 0, 0, 0) \
    X(1, 1, 1, 0, 1) \
    X(2, 2, 2, 0, 4) \
    X(3, 3, 3, 0, 9)
// X(row, path, lm_edge, lm_source)
#define SXB_S0_ROWS(X) \
    X(0, 0, 0, 0) \
    X(1, 1, 1, 0) \
    X(2, 1, 2, 0) \
    X(3, 1, 3, 0) \
    X(4, 2, 4, 0) \
    X(5, 2, 5, 0) \
    X(6, 2, 6, 0) \
    X(7, 2, 7, 0) \
    X(8, 2, 8, 0) \
    X(9, 3, 9, 0) \
    X(10, 3, 10, 0) \
    X(11, 3, 11, 0) \
    X(12, 3, 12, 0) \
    X(13, 3, 13, 0) \
    X(14, 3, 14, 0) \
    X(15, 3, 15, 0)
// X(term, row, lme): coefficient values live in constant memory, indexed by term
#define SXB_S0_TERMS(X) \
    X(0, 0, 0) \
    X(1, 1, 1) \
    X(2, 2, 2) \
    X(3, 3, 3) \
    X(4, 4, 4) \
    X(5, 5, 5) \
    X(6, 6, 6) \
    X(7, 7, 7) \
    X(8, 8, 8) \
    X(9, 9, 9) \
    X(10, 10, 10) \
    X(11, 11, 11) \
    X(12, 12, 12) \
    X(13, 13, 13) \
    X(14, 14, 14) \
    X(15, 15, 15)
// this library's own derivation of the coupling coefficients, by term (a model file carries its own)
#define SXB_S0_DEFAULT_CG {1.0f, 1.0f, 0.9999999999999997f, 0.9999999999999994f, 1.0f, 1.0000000000000004f, 1.0000000000000013f, 1.0000000000000009f, 1.0000000000000013f, 1.0f, 1.0000000000000002f, 1.0000000000000013f, 0.9999999999999994f, 0.999999999999999f, 0.9999999999999997f, 1.0000000000000002f}
#define SXB_S0_M0_NUM_TERMS 94
#define SXB_S0_M0_OFFSETS {0, 94}
// X1(out, term, a)  X2(out, term, a, b)  X3(out, term, a, b, c)
#define SXB_S0_M0_TERMS(X1, X2, X3) \
    X1(0, 0, 0) \
    X2(0, 1, 0, 0) \
    X2(0, 2, 1, 1) \
    X2(0, 3, 2, 2) \
    X2(0, 4, 3, 3) \
    X2(0, 5, 4, 4) \
    X2(0, 6, 5, 5) \
    X2(0, 7, 6, 6) \
    X2(0, 8, 7, 7) \
    X2(0, 9, 8, 8) \
    X2(0, 10, 9, 9) \
    X2(0, 11, 10, 10) \
    X2(0, 12, 11, 11) \
    X2(0, 13, 12, 12) \
    X2(0, 14, 13, 13) \
    X2(0, 15, 14, 14) \
    X2(0, 16, 15, 15) \
    X3(0, 17, 0, 0, 0) \
    X3(0, 18, 0, 1, 1) \
    X3(0, 19, 0, 2, 2) \
    X3(0, 20, 0, 3, 3) \
    X3(0, 21, 0, 4, 4) \
    X3(0, 22, 0, 5, 5) \
    X3(0, 23, 0, 6, 6) \
    X3(0, 24, 0, 7, 7) \
    X3(0, 25, 0, 8, 8) \
    X3(0, 26, 0, 9, 9) \
    X3(0, 27, 0, 10, 10) \
    X3(0, 28, 0, 11, 11) \
    X3(0, 29, 0, 12, 12) \
    X3(0, 30, 0, 13, 13) \
    X3(0, 31, 0, 14, 14) \
    X3(0, 32, 0, 15, 15) \
    X3(0, 33, 1, 1, 6) \
    X3(0, 34, 1, 1, 8) \
    X3(0, 35, 1, 2, 5) \
    X3(0, 36, 1, 3, 4) \
    X3(0, 37, 1, 4, 13) \
    X3(0, 38, 1, 4, 15) \
    X3(0, 39, 1, 5, 12) \
    X3(0, 40, 1, 5, 14) \
    X3(0, 41, 1, 6, 11) \
    X3(0, 42, 1, 7, 10) \
    X3(0, 43, 1, 8, 9) \
    X3(0, 44, 1, 8, 11) \
    X3(0, 45, 2, 2, 6) \
    X3(0, 46, 2, 3, 7) \
    X3(0, 47, 2, 4, 10) \
    X3(0, 48, 2, 5, 11) \
    X3(0, 49, 2, 6, 12) \
    X3(0, 50, 2, 7, 13) \
    X3(0, 51, 2, 8, 14) \
    X3(0, 52, 3, 3, 6) \
    X3(0, 53, 3, 3, 8) \
    X3(0, 54, 3, 4, 9) \
    X3(0, 55, 3, 4, 11) \
    X3(0, 56, 3, 5, 10) \
    X3(0, 57, 3, 6, 13) \
    X3(0, 58, 3, 7, 12) \
    X3(0, 59, 3, 7, 14) \
    X3(0, 60, 3, 8, 13) \
    X3(0, 61, 3, 8, 15) \
    X3(0, 62, 4, 4, 6) \
    X3(0, 63, 4, 5, 7) \
    X3(0, 64, 4, 9, 13) \
    X3(0, 65, 4, 10, 12) \
    X3(0, 66, 4, 11, 13) \
    X3(0, 67, 4, 11, 15) \
    X3(0, 68, 5, 5, 6) \
    X3(0, 69, 5, 5, 8) \
    X3(0, 70, 5, 9, 14) \
    X3(0, 71, 5, 10, 13) \
    X3(0, 72, 5, 10, 15) \
    X3(0, 73, 5, 11, 12) \
    X3(0, 74, 5, 11, 14) \
    X3(0, 75, 6, 6, 6) \
    X3(0, 76, 6, 7, 7) \
    X3(0, 77, 6, 8, 8) \
    X3(0, 78, 6, 9, 9) \
    X3(0, 79, 6, 11, 11) \
    X3(0, 80, 6, 12, 12) \
    X3(0, 81, 6, 13, 13) \
    X3(0, 82, 6, 15, 15) \
    X3(0, 83, 7, 7, 8) \
    X3(0, 84, 7, 9, 10) \
    X3(0, 85, 7, 10, 11) \
    X3(0, 86, 7, 12, 13) \
    X3(0, 87, 7, 13, 14) \
    X3(0, 88, 7, 14, 15) \
    X3(0, 89, 8, 9, 11) \
    X3(0, 90, 8, 11, 11) \
    X3(0, 91, 8, 12, 14) \
    X3(0, 92, 8, 13, 13) \
    X3(0, 93, 8, 13, 15)
#define SXB_S0_M1_NUM_TERMS 94
#define SXB_S0_M1_TERMS(X1, X2, X3) \
    X1(0, 0, 0) \
    X2(0, 1, 0, 0) \
    X2(0, 2, 1, 1) \
    X2(0, 3, 2, 2) \
    X2(0, 4, 3, 3) \
    X2(0, 5, 4, 4) \
    X2(0, 6, 5, 5) \
    X2(0, 7, 6, 6) \
    X2(0, 8, 7, 7) \
    X2(0, 9, 8, 8) \
    X2(0, 10, 9, 9) \
    X2(0, 11, 10, 10) \
    X2(0, 12, 11, 11) \
    X2(0, 13, 12, 12) \
    X2(0, 14, 13, 13) \
    X2(0, 15, 14, 14) \
    X2(0, 16, 15, 15) \
    X3(0, 17, 0, 0, 0) \
    X3(0, 18, 0, 1, 1) \
    X3(0, 19, 0, 2, 2) \
    X3(0, 20, 0, 3, 3) \
    X3(0, 21, 0, 4, 4) \
    X3(0, 22, 0, 5, 5) \
    X3(0, 23, 0, 6, 6) \
    X3(0, 24, 0, 7, 7) \
    X3(0, 25, 0, 8, 8) \
    X3(0, 26, 0, 9, 9) \
    X3(0, 27, 0, 10, 10) \
    X3(0, 28, 0, 11, 11) \
    X3(0, 29, 0, 12, 12) \
    X3(0, 30, 0, 13, 13) \
    X3(0, 31, 0, 14, 14) \
    X3(0, 32, 0, 15, 15) \
    X3(0, 33, 1, 1, 6) \
    X3(0, 34, 1, 1, 8) \
    X3(0, 35, 1, 2, 5) \
    X3(0, 36, 1, 3, 4) \
    X3(0, 37, 1, 4, 13) \
    X3(0, 38, 1, 4, 15) \
    X3(0, 39, 1, 5, 12) \
    X3(0, 40, 1, 5, 14) \
    X3(0, 41, 1, 6, 11) \
    X3(0, 42, 1, 7, 10) \
    X3(0, 43, 1, 8, 9) \
    X3(0, 44, 1, 8, 11) \
    X3(0, 45, 2, 2, 6) \
    X3(0, 46, 2, 3, 7) \
    X3(0, 47, 2, 4, 10) \
    X3(0, 48, 2, 5, 11) \
    X3(0, 49, 2, 6, 12) \
    X3(0, 50, 2, 7, 13) \
    X3(0, 51, 2, 8, 14) \
    X3(0, 52, 3, 3, 6) \
    X3(0, 53, 3, 3, 8) \
    X3(0, 54, 3, 4, 9) \
    X3(0, 55, 3, 4, 11) \
    X3(0, 56, 3, 5, 10) \
    X3(0, 57, 3, 6, 13) \
    X3(0, 58, 3, 7, 12) \
    X3(0, 59, 3, 7, 14) \
    X3(0, 60, 3, 8, 13) \
    X3(0, 61, 3, 8, 15) \
    X3(0, 62, 4, 4, 6) \
    X3(0, 63, 4, 5, 7) \
    X3(0, 64, 4, 9, 13) \
    X3(0, 65, 4, 10, 12) \
    X3(0, 66, 4, 11, 13) \
    X3(0, 67, 4, 11, 15) \
    X3(0, 68, 5, 5, 6) \
    X3(0, 69, 5, 5, 8) \
    X3(0, 70, 5, 9, 14) \
    X3(0, 71, 5, 10, 13) \
    X3(0, 72, 5, 10, 15) \
    X3(0, 73, 5, 11, 12) \
    X3(0, 74, 5, 11, 14) \
    X3(0, 75, 6, 6, 6) \
    X3(0, 76, 6, 7, 7) \
    X3(0, 77, 6, 8, 8) \
    X3(0, 78, 6, 9, 9) \
    X3(0, 79, 6, 11, 11) \
    X3(0, 80, 6, 12, 12) \
    X3(0, 81, 6, 13, 13) \
    X3(0, 82, 6, 15, 15) \
    X3(0, 83, 7, 7, 8) \
    X3(0, 84, 7, 9, 10) \
    X3(0, 85, 7, 10, 11) \
    X3(0, 86, 7, 12, 13) \
    X3(0, 87, 7, 13, 14) \
    X3(0, 88, 7, 14, 15) \
    X3(0, 89, 8, 9, 11) \
    X3(0, 90, 8, 11, 11) \
    X3(0, 91, 8, 12, 14) \
    X3(0, 92, 8, 13, 13) \
    X3(0, 93, 8, 13, 15)
#define SXB_S0_M0_FORWARD_BODY \
      o[0] = f2_fma(W(0), x[0], o[0]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); o[0] = f2_fma(p, f2_fma(W(17), x[0], W(1)), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); o[0] = f2_fma(p, f2_mul(W(18), x[1]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); o[0] = f2_fma(p, f2_mul(W(19), x[2]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); o[0] = f2_fma(p, f2_mul(W(20), x[3]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); o[0] = f2_fma(p, f2_mul(W(21), x[4]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); o[0] = f2_fma(p, f2_mul(W(22), x[5]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); o[0] = f2_fma(p, f2_mul(W(23), x[6]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); o[0] = f2_fma(p, f2_mul(W(24), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); o[0] = f2_fma(p, f2_mul(W(25), x[8]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); o[0] = f2_fma(p, f2_mul(W(26), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); o[0] = f2_fma(p, f2_mul(W(27), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); o[0] = f2_fma(p, f2_mul(W(28), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); o[0] = f2_fma(p, f2_mul(W(29), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); o[0] = f2_fma(p, f2_mul(W(30), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); o[0] = f2_fma(p, f2_mul(W(31), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); o[0] = f2_fma(p, f2_mul(W(32), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); o[0] = f2_fma(p, f2_fma(W(34), x[8], f2_fma(W(33), x[6], W(2))), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); o[0] = f2_fma(p, f2_mul(W(35), x[5]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); o[0] = f2_fma(p, f2_mul(W(36), x[4]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); o[0] = f2_fma(p, f2_fma(W(38), x[15], f2_mul(W(37), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); o[0] = f2_fma(p, f2_fma(W(40), x[14], f2_mul(W(39), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); o[0] = f2_fma(p, f2_mul(W(41), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); o[0] = f2_fma(p, f2_mul(W(42), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); o[0] = f2_fma(p, f2_fma(W(44), x[11], f2_mul(W(43), x[9])), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); o[0] = f2_fma(p, f2_fma(W(45), x[6], W(3)), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); o[0] = f2_fma(p, f2_mul(W(46), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); o[0] = f2_fma(p, f2_mul(W(47), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); o[0] = f2_fma(p, f2_mul(W(48), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); o[0] = f2_fma(p, f2_mul(W(49), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); o[0] = f2_fma(p, f2_mul(W(50), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); o[0] = f2_fma(p, f2_mul(W(51), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); o[0] = f2_fma(p, f2_fma(W(53), x[8], f2_fma(W(52), x[6], W(4))), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); o[0] = f2_fma(p, f2_fma(W(55), x[11], f2_mul(W(54), x[9])), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); o[0] = f2_fma(p, f2_mul(W(56), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); o[0] = f2_fma(p, f2_mul(W(57), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); o[0] = f2_fma(p, f2_fma(W(59), x[14], f2_mul(W(58), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); o[0] = f2_fma(p, f2_fma(W(61), x[15], f2_mul(W(60), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); o[0] = f2_fma(p, f2_fma(W(62), x[6], W(5)), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); o[0] = f2_fma(p, f2_mul(W(63), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); o[0] = f2_fma(p, f2_mul(W(64), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); o[0] = f2_fma(p, f2_mul(W(65), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); o[0] = f2_fma(p, f2_fma(W(67), x[15], f2_mul(W(66), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); o[0] = f2_fma(p, f2_fma(W(69), x[8], f2_fma(W(68), x[6], W(6))), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); o[0] = f2_fma(p, f2_mul(W(70), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); o[0] = f2_fma(p, f2_fma(W(72), x[15], f2_mul(W(71), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); o[0] = f2_fma(p, f2_fma(W(74), x[14], f2_mul(W(73), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); o[0] = f2_fma(p, f2_fma(W(75), x[6], W(7)), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); o[0] = f2_fma(p, f2_mul(W(76), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); o[0] = f2_fma(p, f2_mul(W(77), x[8]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); o[0] = f2_fma(p, f2_mul(W(78), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); o[0] = f2_fma(p, f2_mul(W(79), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); o[0] = f2_fma(p, f2_mul(W(80), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); o[0] = f2_fma(p, f2_mul(W(81), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); o[0] = f2_fma(p, f2_mul(W(82), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); o[0] = f2_fma(p, f2_fma(W(83), x[8], W(8)), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); o[0] = f2_fma(p, f2_mul(W(84), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); o[0] = f2_fma(p, f2_mul(W(85), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); o[0] = f2_fma(p, f2_mul(W(86), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); o[0] = f2_fma(p, f2_mul(W(87), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); o[0] = f2_fma(p, f2_mul(W(88), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[8]); o[0] = f2_fma(p, W(9), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); o[0] = f2_fma(p, f2_mul(W(89), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); o[0] = f2_fma(p, f2_mul(W(90), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); o[0] = f2_fma(p, f2_mul(W(91), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); o[0] = f2_fma(p, f2_fma(W(93), x[15], f2_mul(W(92), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[9], x[9]); o[0] = f2_fma(p, W(10), o[0]); } \
      { const unsigned long long p = f2_mul(x[10], x[10]); o[0] = f2_fma(p, W(11), o[0]); } \
      { const unsigned long long p = f2_mul(x[11], x[11]); o[0] = f2_fma(p, W(12), o[0]); } \
      { const unsigned long long p = f2_mul(x[12], x[12]); o[0] = f2_fma(p, W(13), o[0]); } \
      { const unsigned long long p = f2_mul(x[13], x[13]); o[0] = f2_fma(p, W(14), o[0]); } \
      { const unsigned long long p = f2_mul(x[14], x[14]); o[0] = f2_fma(p, W(15), o[0]); } \
      { const unsigned long long p = f2_mul(x[15], x[15]); o[0] = f2_fma(p, W(16), o[0]); }
#define SXB_S0_M0_REVERSE_BODY \
      g[0] = f2_fma(W(0), adj[0], g[0]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); unsigned long long v; v = f2_mul(W(1), adj[0]); { const unsigned long long s = f2_mul(W(17), adj[0]); g[0] = f2_fma(s, p, g[0]); v = f2_fma(s, x[0], v); } g[0] = f2_fma(v, x[0], g[0]); g[0] = f2_fma(v, x[0], g[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); unsigned long long v; { const unsigned long long s = f2_mul(W(18), adj[0]); g[1] = f2_fma(s, p, g[1]); v = f2_mul(s, x[1]); } g[0] = f2_fma(v, x[1], g[0]); g[1] = f2_fma(v, x[0], g[1]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(19), adj[0]); g[2] = f2_fma(s, p, g[2]); v = f2_mul(s, x[2]); } g[0] = f2_fma(v, x[2], g[0]); g[2] = f2_fma(v, x[0], g[2]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(20), adj[0]); g[3] = f2_fma(s, p, g[3]); v = f2_mul(s, x[3]); } g[0] = f2_fma(v, x[3], g[0]); g[3] = f2_fma(v, x[0], g[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(21), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } g[0] = f2_fma(v, x[4], g[0]); g[4] = f2_fma(v, x[0], g[4]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(22), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } g[0] = f2_fma(v, x[5], g[0]); g[5] = f2_fma(v, x[0], g[5]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(23), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_mul(s, x[6]); } g[0] = f2_fma(v, x[6], g[0]); g[6] = f2_fma(v, x[0], g[6]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(24), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[0] = f2_fma(v, x[7], g[0]); g[7] = f2_fma(v, x[0], g[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(25), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } g[0] = f2_fma(v, x[8], g[0]); g[8] = f2_fma(v, x[0], g[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(26), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[0] = f2_fma(v, x[9], g[0]); g[9] = f2_fma(v, x[0], g[9]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(27), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[0] = f2_fma(v, x[10], g[0]); g[10] = f2_fma(v, x[0], g[10]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(28), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[0] = f2_fma(v, x[11], g[0]); g[11] = f2_fma(v, x[0], g[11]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(29), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[0] = f2_fma(v, x[12], g[0]); g[12] = f2_fma(v, x[0], g[12]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(30), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[0] = f2_fma(v, x[13], g[0]); g[13] = f2_fma(v, x[0], g[13]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(31), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[0] = f2_fma(v, x[14], g[0]); g[14] = f2_fma(v, x[0], g[14]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(32), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[0] = f2_fma(v, x[15], g[0]); g[15] = f2_fma(v, x[0], g[15]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); unsigned long long v; v = f2_mul(W(2), adj[0]); { const unsigned long long s = f2_mul(W(33), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(34), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[1] = f2_fma(v, x[1], g[1]); g[1] = f2_fma(v, x[1], g[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(35), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } g[1] = f2_fma(v, x[2], g[1]); g[2] = f2_fma(v, x[1], g[2]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(36), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } g[1] = f2_fma(v, x[3], g[1]); g[3] = f2_fma(v, x[1], g[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(37), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(38), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[4], g[1]); g[4] = f2_fma(v, x[1], g[4]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(39), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(40), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[5], g[1]); g[5] = f2_fma(v, x[1], g[5]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(41), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[1] = f2_fma(v, x[6], g[1]); g[6] = f2_fma(v, x[1], g[6]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(42), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[1] = f2_fma(v, x[7], g[1]); g[7] = f2_fma(v, x[1], g[7]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(43), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(44), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[1] = f2_fma(v, x[8], g[1]); g[8] = f2_fma(v, x[1], g[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); unsigned long long v; v = f2_mul(W(3), adj[0]); { const unsigned long long s = f2_mul(W(45), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[2] = f2_fma(v, x[2], g[2]); g[2] = f2_fma(v, x[2], g[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(46), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[2] = f2_fma(v, x[3], g[2]); g[3] = f2_fma(v, x[2], g[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(47), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[2] = f2_fma(v, x[4], g[2]); g[4] = f2_fma(v, x[2], g[4]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(48), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[2] = f2_fma(v, x[5], g[2]); g[5] = f2_fma(v, x[2], g[5]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(49), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[2] = f2_fma(v, x[6], g[2]); g[6] = f2_fma(v, x[2], g[6]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(50), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[2] = f2_fma(v, x[7], g[2]); g[7] = f2_fma(v, x[2], g[7]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(51), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[2] = f2_fma(v, x[8], g[2]); g[8] = f2_fma(v, x[2], g[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); unsigned long long v; v = f2_mul(W(4), adj[0]); { const unsigned long long s = f2_mul(W(52), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(53), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[3] = f2_fma(v, x[3], g[3]); g[3] = f2_fma(v, x[3], g[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(54), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(55), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[3] = f2_fma(v, x[4], g[3]); g[4] = f2_fma(v, x[3], g[4]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(56), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[3] = f2_fma(v, x[5], g[3]); g[5] = f2_fma(v, x[3], g[5]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(57), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[3] = f2_fma(v, x[6], g[3]); g[6] = f2_fma(v, x[3], g[6]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(58), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(59), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[3] = f2_fma(v, x[7], g[3]); g[7] = f2_fma(v, x[3], g[7]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(60), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(61), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[8], g[3]); g[8] = f2_fma(v, x[3], g[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); unsigned long long v; v = f2_mul(W(5), adj[0]); { const unsigned long long s = f2_mul(W(62), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[4] = f2_fma(v, x[4], g[4]); g[4] = f2_fma(v, x[4], g[4]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(63), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[4] = f2_fma(v, x[5], g[4]); g[5] = f2_fma(v, x[4], g[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(64), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[4] = f2_fma(v, x[9], g[4]); g[9] = f2_fma(v, x[4], g[9]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(65), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[4] = f2_fma(v, x[10], g[4]); g[10] = f2_fma(v, x[4], g[10]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(66), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(67), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[11], g[4]); g[11] = f2_fma(v, x[4], g[11]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); unsigned long long v; v = f2_mul(W(6), adj[0]); { const unsigned long long s = f2_mul(W(68), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(69), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[5] = f2_fma(v, x[5], g[5]); g[5] = f2_fma(v, x[5], g[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(70), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[5] = f2_fma(v, x[9], g[5]); g[9] = f2_fma(v, x[5], g[9]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(71), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(72), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[10], g[5]); g[10] = f2_fma(v, x[5], g[10]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(73), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(74), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[11], g[5]); g[11] = f2_fma(v, x[5], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); unsigned long long v; v = f2_mul(W(7), adj[0]); { const unsigned long long s = f2_mul(W(75), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[6] = f2_fma(v, x[6], g[6]); g[6] = f2_fma(v, x[6], g[6]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(76), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[6] = f2_fma(v, x[7], g[6]); g[7] = f2_fma(v, x[6], g[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(77), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } g[6] = f2_fma(v, x[8], g[6]); g[8] = f2_fma(v, x[6], g[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(78), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[6] = f2_fma(v, x[9], g[6]); g[9] = f2_fma(v, x[6], g[9]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(79), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[6] = f2_fma(v, x[11], g[6]); g[11] = f2_fma(v, x[6], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(80), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[6] = f2_fma(v, x[12], g[6]); g[12] = f2_fma(v, x[6], g[12]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(81), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[6] = f2_fma(v, x[13], g[6]); g[13] = f2_fma(v, x[6], g[13]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(82), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[6] = f2_fma(v, x[15], g[6]); g[15] = f2_fma(v, x[6], g[15]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); unsigned long long v; v = f2_mul(W(8), adj[0]); { const unsigned long long s = f2_mul(W(83), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[7] = f2_fma(v, x[7], g[7]); g[7] = f2_fma(v, x[7], g[7]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(84), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[7] = f2_fma(v, x[9], g[7]); g[9] = f2_fma(v, x[7], g[9]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(85), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[7] = f2_fma(v, x[10], g[7]); g[10] = f2_fma(v, x[7], g[10]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(86), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[7] = f2_fma(v, x[12], g[7]); g[12] = f2_fma(v, x[7], g[12]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(87), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[7] = f2_fma(v, x[13], g[7]); g[13] = f2_fma(v, x[7], g[13]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(88), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[7] = f2_fma(v, x[14], g[7]); g[14] = f2_fma(v, x[7], g[14]); } \
      { unsigned long long v; v = f2_mul(W(9), adj[0]); g[8] = f2_fma(v, x[8], g[8]); g[8] = f2_fma(v, x[8], g[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(89), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[8] = f2_fma(v, x[9], g[8]); g[9] = f2_fma(v, x[8], g[9]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(90), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[8] = f2_fma(v, x[11], g[8]); g[11] = f2_fma(v, x[8], g[11]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(91), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[8] = f2_fma(v, x[12], g[8]); g[12] = f2_fma(v, x[8], g[12]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(92), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(93), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[13], g[8]); g[13] = f2_fma(v, x[8], g[13]); } \
      { unsigned long long v; v = f2_mul(W(10), adj[0]); g[9] = f2_fma(v, x[9], g[9]); g[9] = f2_fma(v, x[9], g[9]); } \
      { unsigned long long v; v = f2_mul(W(11), adj[0]); g[10] = f2_fma(v, x[10], g[10]); g[10] = f2_fma(v, x[10], g[10]); } \
      { unsigned long long v; v = f2_mul(W(12), adj[0]); g[11] = f2_fma(v, x[11], g[11]); g[11] = f2_fma(v, x[11], g[11]); } \
      { unsigned long long v; v = f2_mul(W(13), adj[0]); g[12] = f2_fma(v, x[12], g[12]); g[12] = f2_fma(v, x[12], g[12]); } \
      { unsigned long long v; v = f2_mul(W(14), adj[0]); g[13] = f2_fma(v, x[13], g[13]); g[13] = f2_fma(v, x[13], g[13]); } \
      { unsigned long long v; v = f2_mul(W(15), adj[0]); g[14] = f2_fma(v, x[14], g[14]); g[14] = f2_fma(v, x[14], g[14]); } \
      { unsigned long long v; v = f2_mul(W(16), adj[0]); g[15] = f2_fma(v, x[15], g[15]); g[15] = f2_fma(v, x[15], g[15]); }
#define SXB_S0_M1_FORWARD_BODY \
      o[0] = f2_fma(W(0), x[0], o[0]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); o[0] = f2_fma(p, f2_fma(W(17), x[0], W(1)), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); o[0] = f2_fma(p, f2_mul(W(18), x[1]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); o[0] = f2_fma(p, f2_mul(W(19), x[2]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); o[0] = f2_fma(p, f2_mul(W(20), x[3]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); o[0] = f2_fma(p, f2_mul(W(21), x[4]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); o[0] = f2_fma(p, f2_mul(W(22), x[5]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); o[0] = f2_fma(p, f2_mul(W(23), x[6]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); o[0] = f2_fma(p, f2_mul(W(24), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); o[0] = f2_fma(p, f2_mul(W(25), x[8]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); o[0] = f2_fma(p, f2_mul(W(26), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); o[0] = f2_fma(p, f2_mul(W(27), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); o[0] = f2_fma(p, f2_mul(W(28), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); o[0] = f2_fma(p, f2_mul(W(29), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); o[0] = f2_fma(p, f2_mul(W(30), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); o[0] = f2_fma(p, f2_mul(W(31), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); o[0] = f2_fma(p, f2_mul(W(32), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); o[0] = f2_fma(p, f2_fma(W(34), x[8], f2_fma(W(33), x[6], W(2))), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); o[0] = f2_fma(p, f2_mul(W(35), x[5]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); o[0] = f2_fma(p, f2_mul(W(36), x[4]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); o[0] = f2_fma(p, f2_fma(W(38), x[15], f2_mul(W(37), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); o[0] = f2_fma(p, f2_fma(W(40), x[14], f2_mul(W(39), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); o[0] = f2_fma(p, f2_mul(W(41), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); o[0] = f2_fma(p, f2_mul(W(42), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); o[0] = f2_fma(p, f2_fma(W(44), x[11], f2_mul(W(43), x[9])), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); o[0] = f2_fma(p, f2_fma(W(45), x[6], W(3)), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); o[0] = f2_fma(p, f2_mul(W(46), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); o[0] = f2_fma(p, f2_mul(W(47), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); o[0] = f2_fma(p, f2_mul(W(48), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); o[0] = f2_fma(p, f2_mul(W(49), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); o[0] = f2_fma(p, f2_mul(W(50), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); o[0] = f2_fma(p, f2_mul(W(51), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); o[0] = f2_fma(p, f2_fma(W(53), x[8], f2_fma(W(52), x[6], W(4))), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); o[0] = f2_fma(p, f2_fma(W(55), x[11], f2_mul(W(54), x[9])), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); o[0] = f2_fma(p, f2_mul(W(56), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); o[0] = f2_fma(p, f2_mul(W(57), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); o[0] = f2_fma(p, f2_fma(W(59), x[14], f2_mul(W(58), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); o[0] = f2_fma(p, f2_fma(W(61), x[15], f2_mul(W(60), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); o[0] = f2_fma(p, f2_fma(W(62), x[6], W(5)), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); o[0] = f2_fma(p, f2_mul(W(63), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); o[0] = f2_fma(p, f2_mul(W(64), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); o[0] = f2_fma(p, f2_mul(W(65), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); o[0] = f2_fma(p, f2_fma(W(67), x[15], f2_mul(W(66), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); o[0] = f2_fma(p, f2_fma(W(69), x[8], f2_fma(W(68), x[6], W(6))), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); o[0] = f2_fma(p, f2_mul(W(70), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); o[0] = f2_fma(p, f2_fma(W(72), x[15], f2_mul(W(71), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); o[0] = f2_fma(p, f2_fma(W(74), x[14], f2_mul(W(73), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); o[0] = f2_fma(p, f2_fma(W(75), x[6], W(7)), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); o[0] = f2_fma(p, f2_mul(W(76), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); o[0] = f2_fma(p, f2_mul(W(77), x[8]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); o[0] = f2_fma(p, f2_mul(W(78), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); o[0] = f2_fma(p, f2_mul(W(79), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); o[0] = f2_fma(p, f2_mul(W(80), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); o[0] = f2_fma(p, f2_mul(W(81), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); o[0] = f2_fma(p, f2_mul(W(82), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); o[0] = f2_fma(p, f2_fma(W(83), x[8], W(8)), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); o[0] = f2_fma(p, f2_mul(W(84), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); o[0] = f2_fma(p, f2_mul(W(85), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); o[0] = f2_fma(p, f2_mul(W(86), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); o[0] = f2_fma(p, f2_mul(W(87), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); o[0] = f2_fma(p, f2_mul(W(88), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[8]); o[0] = f2_fma(p, W(9), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); o[0] = f2_fma(p, f2_mul(W(89), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); o[0] = f2_fma(p, f2_mul(W(90), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); o[0] = f2_fma(p, f2_mul(W(91), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); o[0] = f2_fma(p, f2_fma(W(93), x[15], f2_mul(W(92), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[9], x[9]); o[0] = f2_fma(p, W(10), o[0]); } \
      { const unsigned long long p = f2_mul(x[10], x[10]); o[0] = f2_fma(p, W(11), o[0]); } \
      { const unsigned long long p = f2_mul(x[11], x[11]); o[0] = f2_fma(p, W(12), o[0]); } \
      { const unsigned long long p = f2_mul(x[12], x[12]); o[0] = f2_fma(p, W(13), o[0]); } \
      { const unsigned long long p = f2_mul(x[13], x[13]); o[0] = f2_fma(p, W(14), o[0]); } \
      { const unsigned long long p = f2_mul(x[14], x[14]); o[0] = f2_fma(p, W(15), o[0]); } \
      { const unsigned long long p = f2_mul(x[15], x[15]); o[0] = f2_fma(p, W(16), o[0]); }
#define SXB_S0_M1_REVERSE_BODY \
      g[0] = f2_fma(W(0), adj[0], g[0]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); unsigned long long v; v = f2_mul(W(1), adj[0]); { const unsigned long long s = f2_mul(W(17), adj[0]); g[0] = f2_fma(s, p, g[0]); v = f2_fma(s, x[0], v); } g[0] = f2_fma(v, x[0], g[0]); g[0] = f2_fma(v, x[0], g[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); unsigned long long v; { const unsigned long long s = f2_mul(W(18), adj[0]); g[1] = f2_fma(s, p, g[1]); v = f2_mul(s, x[1]); } g[0] = f2_fma(v, x[1], g[0]); g[1] = f2_fma(v, x[0], g[1]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(19), adj[0]); g[2] = f2_fma(s, p, g[2]); v = f2_mul(s, x[2]); } g[0] = f2_fma(v, x[2], g[0]); g[2] = f2_fma(v, x[0], g[2]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(20), adj[0]); g[3] = f2_fma(s, p, g[3]); v = f2_mul(s, x[3]); } g[0] = f2_fma(v, x[3], g[0]); g[3] = f2_fma(v, x[0], g[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(21), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } g[0] = f2_fma(v, x[4], g[0]); g[4] = f2_fma(v, x[0], g[4]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(22), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } g[0] = f2_fma(v, x[5], g[0]); g[5] = f2_fma(v, x[0], g[5]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(23), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_mul(s, x[6]); } g[0] = f2_fma(v, x[6], g[0]); g[6] = f2_fma(v, x[0], g[6]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(24), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[0] = f2_fma(v, x[7], g[0]); g[7] = f2_fma(v, x[0], g[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(25), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } g[0] = f2_fma(v, x[8], g[0]); g[8] = f2_fma(v, x[0], g[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(26), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[0] = f2_fma(v, x[9], g[0]); g[9] = f2_fma(v, x[0], g[9]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(27), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[0] = f2_fma(v, x[10], g[0]); g[10] = f2_fma(v, x[0], g[10]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(28), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[0] = f2_fma(v, x[11], g[0]); g[11] = f2_fma(v, x[0], g[11]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(29), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[0] = f2_fma(v, x[12], g[0]); g[12] = f2_fma(v, x[0], g[12]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(30), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[0] = f2_fma(v, x[13], g[0]); g[13] = f2_fma(v, x[0], g[13]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(31), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[0] = f2_fma(v, x[14], g[0]); g[14] = f2_fma(v, x[0], g[14]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(32), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[0] = f2_fma(v, x[15], g[0]); g[15] = f2_fma(v, x[0], g[15]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); unsigned long long v; v = f2_mul(W(2), adj[0]); { const unsigned long long s = f2_mul(W(33), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(34), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[1] = f2_fma(v, x[1], g[1]); g[1] = f2_fma(v, x[1], g[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(35), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } g[1] = f2_fma(v, x[2], g[1]); g[2] = f2_fma(v, x[1], g[2]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(36), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } g[1] = f2_fma(v, x[3], g[1]); g[3] = f2_fma(v, x[1], g[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(37), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(38), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[4], g[1]); g[4] = f2_fma(v, x[1], g[4]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(39), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(40), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[5], g[1]); g[5] = f2_fma(v, x[1], g[5]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(41), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[1] = f2_fma(v, x[6], g[1]); g[6] = f2_fma(v, x[1], g[6]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(42), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[1] = f2_fma(v, x[7], g[1]); g[7] = f2_fma(v, x[1], g[7]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(43), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(44), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[1] = f2_fma(v, x[8], g[1]); g[8] = f2_fma(v, x[1], g[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); unsigned long long v; v = f2_mul(W(3), adj[0]); { const unsigned long long s = f2_mul(W(45), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[2] = f2_fma(v, x[2], g[2]); g[2] = f2_fma(v, x[2], g[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(46), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[2] = f2_fma(v, x[3], g[2]); g[3] = f2_fma(v, x[2], g[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(47), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[2] = f2_fma(v, x[4], g[2]); g[4] = f2_fma(v, x[2], g[4]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(48), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[2] = f2_fma(v, x[5], g[2]); g[5] = f2_fma(v, x[2], g[5]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(49), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[2] = f2_fma(v, x[6], g[2]); g[6] = f2_fma(v, x[2], g[6]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(50), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[2] = f2_fma(v, x[7], g[2]); g[7] = f2_fma(v, x[2], g[7]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(51), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[2] = f2_fma(v, x[8], g[2]); g[8] = f2_fma(v, x[2], g[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); unsigned long long v; v = f2_mul(W(4), adj[0]); { const unsigned long long s = f2_mul(W(52), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(53), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[3] = f2_fma(v, x[3], g[3]); g[3] = f2_fma(v, x[3], g[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(54), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(55), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[3] = f2_fma(v, x[4], g[3]); g[4] = f2_fma(v, x[3], g[4]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(56), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[3] = f2_fma(v, x[5], g[3]); g[5] = f2_fma(v, x[3], g[5]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(57), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[3] = f2_fma(v, x[6], g[3]); g[6] = f2_fma(v, x[3], g[6]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(58), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(59), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[3] = f2_fma(v, x[7], g[3]); g[7] = f2_fma(v, x[3], g[7]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(60), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(61), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[8], g[3]); g[8] = f2_fma(v, x[3], g[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); unsigned long long v; v = f2_mul(W(5), adj[0]); { const unsigned long long s = f2_mul(W(62), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[4] = f2_fma(v, x[4], g[4]); g[4] = f2_fma(v, x[4], g[4]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(63), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[4] = f2_fma(v, x[5], g[4]); g[5] = f2_fma(v, x[4], g[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(64), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[4] = f2_fma(v, x[9], g[4]); g[9] = f2_fma(v, x[4], g[9]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(65), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[4] = f2_fma(v, x[10], g[4]); g[10] = f2_fma(v, x[4], g[10]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(66), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(67), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[11], g[4]); g[11] = f2_fma(v, x[4], g[11]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); unsigned long long v; v = f2_mul(W(6), adj[0]); { const unsigned long long s = f2_mul(W(68), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(69), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[5] = f2_fma(v, x[5], g[5]); g[5] = f2_fma(v, x[5], g[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(70), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[5] = f2_fma(v, x[9], g[5]); g[9] = f2_fma(v, x[5], g[9]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(71), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(72), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[10], g[5]); g[10] = f2_fma(v, x[5], g[10]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(73), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(74), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[11], g[5]); g[11] = f2_fma(v, x[5], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); unsigned long long v; v = f2_mul(W(7), adj[0]); { const unsigned long long s = f2_mul(W(75), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[6] = f2_fma(v, x[6], g[6]); g[6] = f2_fma(v, x[6], g[6]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(76), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[6] = f2_fma(v, x[7], g[6]); g[7] = f2_fma(v, x[6], g[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(77), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } g[6] = f2_fma(v, x[8], g[6]); g[8] = f2_fma(v, x[6], g[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(78), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[6] = f2_fma(v, x[9], g[6]); g[9] = f2_fma(v, x[6], g[9]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(79), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[6] = f2_fma(v, x[11], g[6]); g[11] = f2_fma(v, x[6], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(80), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[6] = f2_fma(v, x[12], g[6]); g[12] = f2_fma(v, x[6], g[12]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(81), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[6] = f2_fma(v, x[13], g[6]); g[13] = f2_fma(v, x[6], g[13]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(82), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[6] = f2_fma(v, x[15], g[6]); g[15] = f2_fma(v, x[6], g[15]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); unsigned long long v; v = f2_mul(W(8), adj[0]); { const unsigned long long s = f2_mul(W(83), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[7] = f2_fma(v, x[7], g[7]); g[7] = f2_fma(v, x[7], g[7]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(84), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[7] = f2_fma(v, x[9], g[7]); g[9] = f2_fma(v, x[7], g[9]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(85), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[7] = f2_fma(v, x[10], g[7]); g[10] = f2_fma(v, x[7], g[10]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(86), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[7] = f2_fma(v, x[12], g[7]); g[12] = f2_fma(v, x[7], g[12]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(87), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[7] = f2_fma(v, x[13], g[7]); g[13] = f2_fma(v, x[7], g[13]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(88), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[7] = f2_fma(v, x[14], g[7]); g[14] = f2_fma(v, x[7], g[14]); } \
      { unsigned long long v; v = f2_mul(W(9), adj[0]); g[8] = f2_fma(v, x[8], g[8]); g[8] = f2_fma(v, x[8], g[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(89), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[8] = f2_fma(v, x[9], g[8]); g[9] = f2_fma(v, x[8], g[9]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(90), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[8] = f2_fma(v, x[11], g[8]); g[11] = f2_fma(v, x[8], g[11]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(91), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[8] = f2_fma(v, x[12], g[8]); g[12] = f2_fma(v, x[8], g[12]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(92), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(93), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[13], g[8]); g[13] = f2_fma(v, x[8], g[13]); } \
      { unsigned long long v; v = f2_mul(W(10), adj[0]); g[9] = f2_fma(v, x[9], g[9]); g[9] = f2_fma(v, x[9], g[9]); } \
      { unsigned long long v; v = f2_mul(W(11), adj[0]); g[10] = f2_fma(v, x[10], g[10]); g[10] = f2_fma(v, x[10], g[10]); } \
      { unsigned long long v; v = f2_mul(W(12), adj[0]); g[11] = f2_fma(v, x[11], g[11]); g[11] = f2_fma(v, x[11], g[11]); } \
      { unsigned long long v; v = f2_mul(W(13), adj[0]); g[12] = f2_fma(v, x[12], g[12]); g[12] = f2_fma(v, x[12], g[12]); } \
      { unsigned long long v; v = f2_mul(W(14), adj[0]); g[13] = f2_fma(v, x[13], g[13]); g[13] = f2_fma(v, x[13], g[13]); } \
      { unsigned long long v; v = f2_mul(W(15), adj[0]); g[14] = f2_fma(v, x[14], g[14]); g[14] = f2_fma(v, x[14], g[14]); } \
      { unsigned long long v; v = f2_mul(W(16), adj[0]); g[15] = f2_fma(v, x[15], g[15]); g[15] = f2_fma(v, x[15], g[15]); }
#define SXB_S0_L1_FORWARD_BODY \
    { /* path 0: edge l=0, source l=0 -> l=0 */ \
      const float t0 = R[0] * h[0]; \
      acc[0] = fmaf(t0, y[0], acc[0]); \
    } \
    { /* path 1: edge l=1, source l=0 -> l=1 */ \
      const float t0 = R[1] * h[0]; \
      acc[1] = fmaf(t0, y[1], acc[1]); \
      acc[2] = fmaf(t0, y[2], acc[2]); \
      acc[3] = fmaf(t0, y[3], acc[3]); \
    } \
    { /* path 2: edge l=2, source l=0 -> l=2 */ \
      const float t0 = R[2] * h[0]; \
      acc[4] = fmaf(t0, y[4], acc[4]); \
      acc[5] = fmaf(t0, y[5], acc[5]); \
      acc[6] = fmaf(t0, y[6], acc[6]); \
      acc[7] = fmaf(t0, y[7], acc[7]); \
      acc[8] = fmaf(t0, y[8], acc[8]); \
    } \
    { /* path 3: edge l=3, source l=0 -> l=3 */ \
      const float t0 = R[3] * h[0]; \
      acc[9] = fmaf(t0, y[9], acc[9]); \
      acc[10] = fmaf(t0, y[10], acc[10]); \
      acc[11] = fmaf(t0, y[11], acc[11]); \
      acc[12] = fmaf(t0, y[12], acc[12]); \
      acc[13] = fmaf(t0, y[13], acc[13]); \
      acc[14] = fmaf(t0, y[14], acc[14]); \
      acc[15] = fmaf(t0, y[15], acc[15]); \
    }
#define SXB_S0_L1_REVERSE_BODY \
    { /* path 0: edge l=0, source l=0 -> l=0 */ \
      float yw = 0.0f; \
      const float ry0 = R[0] * y[0]; \
      { const float w = h[0] * adj[0]; \
        ang[0] = fmaf(R[0], w, ang[0]); yw = fmaf(y[0], w, yw); } \
      hadj[0] = fmaf(ry0, adj[0], hadj[0]); \
      radial = fmaf(dR[0], yw, radial); \
    } \
    { /* path 1: edge l=1, source l=0 -> l=1 */ \
      float yw = 0.0f; \
      const float rh0 = R[1] * h[0]; \
      ang[1] = fmaf(rh0, adj[1], ang[1]); \
      ang[2] = fmaf(rh0, adj[2], ang[2]); \
      ang[3] = fmaf(rh0, adj[3], ang[3]); \
      { const float s_ = fmaf(y[3], adj[3], fmaf(y[2], adj[2], y[1] * adj[1])); \
        hadj[0] = fmaf(R[1], s_, hadj[0]); yw = fmaf(h[0], s_, yw); } \
      radial = fmaf(dR[1], yw, radial); \
    } \
    { /* path 2: edge l=2, source l=0 -> l=2 */ \
      float yw = 0.0f; \
      const float rh0 = R[2] * h[0]; \
      ang[4] = fmaf(rh0, adj[4], ang[4]); \
      ang[5] = fmaf(rh0, adj[5], ang[5]); \
      ang[6] = fmaf(rh0, adj[6], ang[6]); \
      ang[7] = fmaf(rh0, adj[7], ang[7]); \
      ang[8] = fmaf(rh0, adj[8], ang[8]); \
      { const float s_ = fmaf(y[8], adj[8], fmaf(y[7], adj[7], fmaf(y[6], adj[6], fmaf(y[5], adj[5], y[4] * adj[4])))); \
        hadj[0] = fmaf(R[2], s_, hadj[0]); yw = fmaf(h[0], s_, yw); } \
      radial = fmaf(dR[2], yw, radial); \
    } \
    { /* path 3: edge l=3, source l=0 -> l=3 */ \
      float yw = 0.0f; \
      const float rh0 = R[3] * h[0]; \
      ang[9] = fmaf(rh0, adj[9], ang[9]); \
      ang[10] = fmaf(rh0, adj[10], ang[10]); \
      ang[11] = fmaf(rh0, adj[11], ang[11]); \
      ang[12] = fmaf(rh0, adj[12], ang[12]); \
      ang[13] = fmaf(rh0, adj[13], ang[13]); \
      ang[14] = fmaf(rh0, adj[14], ang[14]); \
      ang[15] = fmaf(rh0, adj[15], ang[15]); \
      { const float s_ = fmaf(y[15], adj[15], fmaf(y[14], adj[14], fmaf(y[13], adj[13], fmaf(y[12], adj[12], fmaf(y[11], adj[11], fmaf(y[10], adj[10], y[9] * adj[9])))))); \
        hadj[0] = fmaf(R[3], s_, hadj[0]); yw = fmaf(h[0], s_, yw); } \
      radial = fmaf(dR[3], yw, radial); \
    }

// ---- shape S1: edge l_max=3, hidden L_max=1
#define SXB_S1_LMAX 3
#define SXB_S1_HIDDEN_LMAX 1
#define SXB_S1_NUM_LM 16
#define SXB_S1_NUM_HIDDEN 4
#define SXB_S1_NUM_PATHS 10
#define SXB_S1_NUM_ROWS 88
#define SXB_S1_NUM_LME 40
#define SXB_S1_NUM_TERMS 86
// X(path, l_out, l_edge, l_source, first_row)
#define SXB_S1_PATHS(X) \
    X(0, 0, 0, 0, 0) \
    X(1, 0, 1, 1, 1) \
    X(2, 1, 1, 0, 10) \
    X(3, 1, 0, 1, 13) \
    X(4, 1, 2, 1, 16) \
    X(5, 2, 2, 0, 31) \
    X(6, 2, 1, 1, 36) \
    X(7, 2, 3, 1, 45) \
    X(8, 3, 3, 0, 66) \
    X(9, 3, 2, 1, 73)
// X(row, path, lm_edge, lm_source)
#define SXB_S1_ROWS(X) \
    X(0, 0, 0, 0) \
    X(1, 1, 1, 1) \
    X(2, 1, 1, 2) \
    X(3, 1, 1, 3) \
    X(4, 1, 2, 1) \
    X(5, 1, 2, 2) \
    X(6, 1, 2, 3) \
    X(7, 1, 3, 1) \
    X(8, 1, 3, 2) \
    X(9, 1, 3, 3) \
    X(10, 2, 1, 0) \
    X(11, 2, 2, 0) \
    X(12, 2, 3, 0) \
    X(13, 3, 0, 1) \
    X(14, 3, 0, 2) \
    X(15, 3, 0, 3) \
    X(16, 4, 4, 1) \
    X(17, 4, 4, 2) \
    X(18, 4, 4, 3) \
    X(19, 4, 5, 1) \
    X(20, 4, 5, 2) \
    X(21, 4, 5, 3) \
    X(22, 4, 6, 1) \
    X(23, 4, 6, 2) \
    X(24, 4, 6, 3) \
    X(25, 4, 7, 1) \
    X(26, 4, 7, 2) \
    X(27, 4, 7, 3) \
    X(28, 4, 8, 1) \
    X(29, 4, 8, 2) \
    X(30, 4, 8, 3) \
    X(31, 5, 4, 0) \
    X(32, 5, 5, 0) \
    X(33, 5, 6, 0) \
    X(34, 5, 7, 0) \
    X(35, 5, 8, 0) \
    X(36, 6, 1, 1) \
    X(37, 6, 1, 2) \
    X(38, 6, 1, 3) \
    X(39, 6, 2, 1) \
    X(40, 6, 2, 2) \
    X(41, 6, 2, 3) \
    X(42, 6, 3, 1) \
    X(43, 6, 3, 2) \
    X(44, 6, 3, 3) \
    X(45, 7, 9, 1) \
    X(46, 7, 9, 2) \
    X(47, 7, 9, 3) \
    X(48, 7, 10, 1) \
    X(49, 7, 10, 2) \
    X(50, 7, 10, 3) \
    X(51, 7, 11, 1) \
    X(52, 7, 11, 2) \
    X(53, 7, 11, 3) \
    X(54, 7, 12, 1) \
    X(55, 7, 12, 2) \
    X(56, 7, 12, 3) \
    X(57, 7, 13, 1) \
    X(58, 7, 13, 2) \
    X(59, 7, 13, 3) \
    X(60, 7, 14, 1) \
    X(61, 7, 14, 2) \
    X(62, 7, 14, 3) \
    X(63, 7, 15, 1) \
    X(64, 7, 15, 2) \
    X(65, 7, 15, 3) \
    X(66, 8, 9, 0) \
    X(67, 8, 10, 0) \
    X(68, 8, 11, 0) \
    X(69, 8, 12, 0) \
    X(70, 8, 13, 0) \
    X(71, 8, 14, 0) \
    X(72, 8, 15, 0) \
    X(73, 9, 4, 1) \
    X(74, 9, 4, 2) \
    X(75, 9, 4, 3) \
    X(76, 9, 5, 1) \
    X(77, 9, 5, 2) \
    X(78, 9, 5, 3) \
    X(79, 9, 6, 1) \
    X(80, 9, 6, 2) \
    X(81, 9, 6, 3) \
    X(82, 9, 7, 1) \
    X(83, 9, 7, 2) \
    X(84, 9, 7, 3) \
    X(85, 9, 8, 1) \
    X(86, 9, 8, 2) \
    X(87, 9, 8, 3)
// X(term, row, lme): coefficient values live in constant memory, indexed by term
#define SXB_S1_TERMS(X) \
    X(0, 0, 0) \
    X(1, 13, 3) \
    X(2, 14, 6) \
    X(3, 15, 9) \
    X(4, 10, 2) \
    X(5, 1, 1) \
    X(6, 36, 18) \
    X(7, 36, 24) \
    X(8, 37, 15) \
    X(9, 38, 12) \
    X(10, 11, 5) \
    X(11, 39, 15) \
    X(12, 5, 1) \
    X(13, 40, 18) \
    X(14, 41, 21) \
    X(15, 12, 8) \
    X(16, 42, 12) \
    X(17, 43, 21) \
    X(18, 9, 1) \
    X(19, 44, 18) \
    X(20, 44, 24) \
    X(21, 31, 11) \
    X(22, 16, 10) \
    X(23, 73, 35) \
    X(24, 73, 39) \
    X(25, 74, 29) \
    X(26, 18, 4) \
    X(27, 75, 27) \
    X(28, 75, 31) \
    X(29, 32, 14) \
    X(30, 19, 7) \
    X(31, 76, 33) \
    X(32, 76, 37) \
    X(33, 20, 4) \
    X(34, 77, 31) \
    X(35, 78, 29) \
    X(36, 33, 17) \
    X(37, 22, 4) \
    X(38, 79, 31) \
    X(39, 23, 7) \
    X(40, 80, 33) \
    X(41, 24, 10) \
    X(42, 81, 35) \
    X(43, 34, 20) \
    X(44, 82, 29) \
    X(45, 26, 10) \
    X(46, 83, 35) \
    X(47, 27, 7) \
    X(48, 84, 33) \
    X(49, 84, 37) \
    X(50, 35, 23) \
    X(51, 28, 4) \
    X(52, 85, 27) \
    X(53, 85, 31) \
    X(54, 86, 37) \
    X(55, 30, 10) \
    X(56, 87, 35) \
    X(57, 87, 39) \
    X(58, 66, 26) \
    X(59, 45, 25) \
    X(60, 47, 13) \
    X(61, 67, 28) \
    X(62, 48, 22) \
    X(63, 49, 13) \
    X(64, 50, 16) \
    X(65, 68, 30) \
    X(66, 51, 19) \
    X(67, 51, 25) \
    X(68, 52, 16) \
    X(69, 53, 13) \
    X(70, 69, 32) \
    X(71, 54, 16) \
    X(72, 55, 19) \
    X(73, 56, 22) \
    X(74, 70, 34) \
    X(75, 57, 13) \
    X(76, 58, 22) \
    X(77, 59, 19) \
    X(78, 59, 25) \
    X(79, 71, 36) \
    X(80, 60, 16) \
    X(81, 61, 25) \
    X(82, 62, 22) \
    X(83, 72, 38) \
    X(84, 63, 13) \
    X(85, 65, 25)
// this library's own derivation of the coupling coefficients, by term (a model file carries its own)
#define SXB_S1_DEFAULT_CG {1.0f, 1.0f, 0.9999999999999998f, 1.0f, 1.0f, 0.5773502691896257f, 0.40824829046386385f, 0.7071067811865485f, -0.7071067811865476f, -0.7071067811865471f, 0.9999999999999997f, -0.7071067811865471f, 0.5773502691896257f, -0.816496580927727f, -0.7071067811865479f, 0.9999999999999994f, -0.7071067811865478f, -0.7071067811865476f, 0.5773502691896258f, 0.4082482904638637f, -0.7071067811865486f, 1.0f, 0.5477225575051663f, 0.1825741858350547f, 0.7071067811865475f, -0.5773502691896257f, 0.547722557505166f, -0.7071067811865475f, 0.18257418583505564f, 1.0000000000000004f, 0.5477225575051659f, 0.4472135954999578f, 0.577350269189626f, 0.547722557505166f, -0.7302967433402211f, -0.5773502691896253f, 1.0000000000000013f, -0.3162277660168377f, -0.6324555320336763f, 0.6324555320336757f, -0.7745966692414836f, -0.31622776601683755f, -0.6324555320336758f, 1.0000000000000009f, -0.5773502691896265f, 0.547722557505166f, -0.7302967433402215f, 0.5477225575051659f, 0.4472135954999579f, -0.5773502691896257f, 1.0000000000000013f, -0.5477225575051666f, -0.7071067811865475f, -0.1825741858350553f, -0.5773502691896262f, 0.547722557505166f, 0.18257418583505564f, -0.7071067811865474f, 1.0f, 0.5976143046671968f, 0.5976143046671969f, 1.0000000000000002f, 0.48795003647426666f, 0.4879500364742665f, 0.48795003647426605f, 1.0000000000000013f, 0.5345224838248491f, 0.1543033499620919f, 0.6172133998483681f, -0.15430334996209205f, 0.9999999999999994f, -0.3779644730092276f, 0.6546536707079776f, -0.37796447300922775f, 0.999999999999999f, -0.15430334996209197f, 0.6172133998483679f, 0.5345224838248491f, -0.15430334996209194f, 0.9999999999999997f, -0.48795003647426655f, 0.4879500364742668f, 0.4879500364742665f, 1.0000000000000002f, -0.5976143046671967f, 0.5976143046671976f}
#define SXB_S1_M0_NUM_TERMS 422
#define SXB_S1_M0_OFFSETS {0, 94, 212, 304, 422}
// X1(out, term, a)  X2(out, term, a, b)  X3(out, term, a, b, c)
#define SXB_S1_M0_TERMS(X1, X2, X3) \
    X1(0, 0, 0) \
    X1(1, 94, 1) \
    X1(2, 212, 2) \
    X1(3, 304, 3) \
    X2(0, 1, 0, 0) \
    X2(0, 2, 1, 1) \
    X2(0, 3, 2, 2) \
    X2(0, 4, 3, 3) \
    X2(0, 5, 4, 4) \
    X2(0, 6, 5, 5) \
    X2(0, 7, 6, 6) \
    X2(0, 8, 7, 7) \
    X2(0, 9, 8, 8) \
    X2(0, 10, 9, 9) \
    X2(0, 11, 10, 10) \
    X2(0, 12, 11, 11) \
    X2(0, 13, 12, 12) \
    X2(0, 14, 13, 13) \
    X2(0, 15, 14, 14) \
    X2(0, 16, 15, 15) \
    X2(1, 95, 0, 1) \
    X2(1, 96, 1, 6) \
    X2(1, 97, 1, 8) \
    X2(1, 98, 2, 5) \
    X2(1, 99, 3, 4) \
    X2(1, 100, 4, 13) \
    X2(1, 101, 4, 15) \
    X2(1, 102, 5, 12) \
    X2(1, 103, 5, 14) \
    X2(1, 104, 6, 11) \
    X2(1, 105, 7, 10) \
    X2(1, 106, 8, 9) \
    X2(1, 107, 8, 11) \
    X2(2, 213, 0, 2) \
    X2(2, 214, 1, 5) \
    X2(2, 215, 2, 6) \
    X2(2, 216, 3, 7) \
    X2(2, 217, 4, 10) \
    X2(2, 218, 5, 11) \
    X2(2, 219, 6, 12) \
    X2(2, 220, 7, 13) \
    X2(2, 221, 8, 14) \
    X2(3, 305, 0, 3) \
    X2(3, 306, 1, 4) \
    X2(3, 307, 2, 7) \
    X2(3, 308, 3, 6) \
    X2(3, 309, 3, 8) \
    X2(3, 310, 4, 9) \
    X2(3, 311, 4, 11) \
    X2(3, 312, 5, 10) \
    X2(3, 313, 6, 13) \
    X2(3, 314, 7, 12) \
    X2(3, 315, 7, 14) \
    X2(3, 316, 8, 13) \
    X2(3, 317, 8, 15) \
    X3(0, 17, 0, 0, 0) \
    X3(0, 18, 0, 1, 1) \
    X3(0, 19, 0, 2, 2) \
    X3(0, 20, 0, 3, 3) \
    X3(0, 21, 0, 4, 4) \
    X3(0, 22, 0, 5, 5) \
    X3(0, 23, 0, 6, 6) \
    X3(0, 24, 0, 7, 7) \
    X3(0, 25, 0, 8, 8) \
    X3(0, 26, 0, 9, 9) \
    X3(0, 27, 0, 10, 10) \
    X3(0, 28, 0, 11, 11) \
    X3(0, 29, 0, 12, 12) \
    X3(0, 30, 0, 13, 13) \
    X3(0, 31, 0, 14, 14) \
    X3(0, 32, 0, 15, 15) \
    X3(0, 33, 1, 1, 6) \
    X3(0, 34, 1, 1, 8) \
    X3(0, 35, 1, 2, 5) \
    X3(0, 36, 1, 3, 4) \
    X3(0, 37, 1, 4, 13) \
    X3(0, 38, 1, 4, 15) \
    X3(0, 39, 1, 5, 12) \
    X3(0, 40, 1, 5, 14) \
    X3(0, 41, 1, 6, 11) \
    X3(0, 42, 1, 7, 10) \
    X3(0, 43, 1, 8, 9) \
    X3(0, 44, 1, 8, 11) \
    X3(0, 45, 2, 2, 6) \
    X3(0, 46, 2, 3, 7) \
    X3(0, 47, 2, 4, 10) \
    X3(0, 48, 2, 5, 11) \
    X3(0, 49, 2, 6, 12) \
    X3(0, 50, 2, 7, 13) \
    X3(0, 51, 2, 8, 14) \
    X3(0, 52, 3, 3, 6) \
    X3(0, 53, 3, 3, 8) \
    X3(0, 54, 3, 4, 9) \
    X3(0, 55, 3, 4, 11) \
    X3(0, 56, 3, 5, 10) \
    X3(0, 57, 3, 6, 13) \
    X3(0, 58, 3, 7, 12) \
    X3(0, 59, 3, 7, 14) \
    X3(0, 60, 3, 8, 13) \
    X3(0, 61, 3, 8, 15) \
    X3(0, 62, 4, 4, 6) \
    X3(0, 63, 4, 5, 7) \
    X3(0, 64, 4, 9, 13) \
    X3(0, 65, 4, 10, 12) \
    X3(0, 66, 4, 11, 13) \
    X3(0, 67, 4, 11, 15) \
    X3(0, 68, 5, 5, 6) \
    X3(0, 69, 5, 5, 8) \
    X3(0, 70, 5, 9, 14) \
    X3(0, 71, 5, 10, 13) \
    X3(0, 72, 5, 10, 15) \
    X3(0, 73, 5, 11, 12) \
    X3(0, 74, 5, 11, 14) \
    X3(0, 75, 6, 6, 6) \
    X3(0, 76, 6, 7, 7) \
    X3(0, 77, 6, 8, 8) \
    X3(0, 78, 6, 9, 9) \
    X3(0, 79, 6, 11, 11) \
    X3(0, 80, 6, 12, 12) \
    X3(0, 81, 6, 13, 13) \
    X3(0, 82, 6, 15, 15) \
    X3(0, 83, 7, 7, 8) \
    X3(0, 84, 7, 9, 10) \
    X3(0, 85, 7, 10, 11) \
    X3(0, 86, 7, 12, 13) \
    X3(0, 87, 7, 13, 14) \
    X3(0, 88, 7, 14, 15) \
    X3(0, 89, 8, 9, 11) \
    X3(0, 90, 8, 11, 11) \
    X3(0, 91, 8, 12, 14) \
    X3(0, 92, 8, 13, 13) \
    X3(0, 93, 8, 13, 15) \
    X3(1, 108, 0, 0, 1) \
    X3(1, 109, 0, 1, 6) \
    X3(1, 110, 0, 1, 8) \
    X3(1, 111, 0, 2, 5) \
    X3(1, 112, 0, 3, 4) \
    X3(1, 113, 0, 4, 13) \
    X3(1, 114, 0, 4, 15) \
    X3(1, 115, 0, 5, 12) \
    X3(1, 116, 0, 5, 14) \
    X3(1, 117, 0, 6, 11) \
    X3(1, 118, 0, 7, 10) \
    X3(1, 119, 0, 8, 9) \
    X3(1, 120, 0, 8, 11) \
    X3(1, 121, 1, 1, 1) \
    X3(1, 122, 1, 1, 9) \
    X3(1, 123, 1, 1, 11) \
    X3(1, 124, 1, 2, 2) \
    X3(1, 125, 1, 2, 12) \
    X3(1, 126, 1, 2, 14) \
    X3(1, 127, 1, 3, 3) \
    X3(1, 128, 1, 3, 13) \
    X3(1, 129, 1, 3, 15) \
    X3(1, 130, 1, 4, 4) \
    X3(1, 131, 1, 5, 5) \
    X3(1, 132, 1, 6, 6) \
    X3(1, 133, 1, 6, 8) \
    X3(1, 134, 1, 7, 7) \
    X3(1, 135, 1, 8, 8) \
    X3(1, 136, 1, 9, 9) \
    X3(1, 137, 1, 9, 11) \
    X3(1, 138, 1, 10, 10) \
    X3(1, 139, 1, 11, 11) \
    X3(1, 140, 1, 12, 12) \
    X3(1, 141, 1, 12, 14) \
    X3(1, 142, 1, 13, 13) \
    X3(1, 143, 1, 13, 15) \
    X3(1, 144, 1, 14, 14) \
    X3(1, 145, 1, 15, 15) \
    X3(1, 146, 2, 2, 11) \
    X3(1, 147, 2, 3, 10) \
    X3(1, 148, 2, 4, 7) \
    X3(1, 149, 2, 5, 6) \
    X3(1, 150, 2, 5, 8) \
    X3(1, 151, 2, 9, 14) \
    X3(1, 152, 2, 10, 13) \
    X3(1, 153, 2, 10, 15) \
    X3(1, 154, 2, 11, 12) \
    X3(1, 155, 2, 11, 14) \
    X3(1, 156, 3, 3, 9) \
    X3(1, 157, 3, 3, 11) \
    X3(1, 158, 3, 4, 6) \
    X3(1, 159, 3, 4, 8) \
    X3(1, 160, 3, 5, 7) \
    X3(1, 161, 3, 9, 13) \
    X3(1, 162, 3, 9, 15) \
    X3(1, 163, 3, 10, 12) \
    X3(1, 164, 3, 10, 14) \
    X3(1, 165, 3, 11, 13) \
    X3(1, 166, 3, 11, 15) \
    X3(1, 167, 4, 4, 9) \
    X3(1, 168, 4, 4, 11) \
    X3(1, 169, 4, 5, 10) \
    X3(1, 170, 4, 6, 13) \
    X3(1, 171, 4, 6, 15) \
    X3(1, 172, 4, 7, 12) \
    X3(1, 173, 4, 7, 14) \
    X3(1, 174, 4, 8, 13) \
    X3(1, 175, 4, 8, 15) \
    X3(1, 176, 5, 5, 9) \
    X3(1, 177, 5, 5, 11) \
    X3(1, 178, 5, 6, 12) \
    X3(1, 179, 5, 6, 14) \
    X3(1, 180, 5, 7, 13) \
    X3(1, 181, 5, 7, 15) \
    X3(1, 182, 5, 8, 12) \
    X3(1, 183, 5, 8, 14) \
    X3(1, 184, 6, 6, 11) \
    X3(1, 185, 6, 7, 10) \
    X3(1, 186, 6, 8, 9) \
    X3(1, 187, 6, 8, 11) \
    X3(1, 188, 7, 7, 9) \
    X3(1, 189, 7, 7, 11) \
    X3(1, 190, 7, 8, 10) \
    X3(1, 191, 8, 8, 9) \
    X3(1, 192, 8, 8, 11) \
    X3(1, 193, 9, 9, 11) \
    X3(1, 194, 9, 10, 10) \
    X3(1, 195, 9, 11, 11) \
    X3(1, 196, 9, 12, 14) \
    X3(1, 197, 9, 13, 13) \
    X3(1, 198, 9, 13, 15) \
    X3(1, 199, 9, 14, 14) \
    X3(1, 200, 10, 10, 11) \
    X3(1, 201, 10, 12, 13) \
    X3(1, 202, 10, 12, 15) \
    X3(1, 203, 10, 13, 14) \
    X3(1, 204, 10, 14, 15) \
    X3(1, 205, 11, 11, 11) \
    X3(1, 206, 11, 12, 12) \
    X3(1, 207, 11, 12, 14) \
    X3(1, 208, 11, 13, 13) \
    X3(1, 209, 11, 13, 15) \
    X3(1, 210, 11, 14, 14) \
    X3(1, 211, 11, 15, 15) \
    X3(2, 222, 0, 0, 2) \
    X3(2, 223, 0, 1, 5) \
    X3(2, 224, 0, 2, 6) \
    X3(2, 225, 0, 3, 7) \
    X3(2, 226, 0, 4, 10) \
    X3(2, 227, 0, 5, 11) \
    X3(2, 228, 0, 6, 12) \
    X3(2, 229, 0, 7, 13) \
    X3(2, 230, 0, 8, 14) \
    X3(2, 231, 1, 1, 2) \
    X3(2, 232, 1, 1, 12) \
    X3(2, 233, 1, 1, 14) \
    X3(2, 234, 1, 2, 11) \
    X3(2, 235, 1, 3, 10) \
    X3(2, 236, 1, 4, 7) \
    X3(2, 237, 1, 5, 6) \
    X3(2, 238, 1, 5, 8) \
    X3(2, 239, 1, 9, 14) \
    X3(2, 240, 1, 10, 13) \
    X3(2, 241, 1, 10, 15) \
    X3(2, 242, 1, 11, 12) \
    X3(2, 243, 1, 11, 14) \
    X3(2, 244, 2, 2, 2) \
    X3(2, 245, 2, 2, 12) \
    X3(2, 246, 2, 3, 3) \
    X3(2, 247, 2, 3, 13) \
    X3(2, 248, 2, 4, 4) \
    X3(2, 249, 2, 5, 5) \
    X3(2, 250, 2, 6, 6) \
    X3(2, 251, 2, 7, 7) \
    X3(2, 252, 2, 8, 8) \
    X3(2, 253, 2, 9, 9) \
    X3(2, 254, 2, 10, 10) \
    X3(2, 255, 2, 11, 11) \
    X3(2, 256, 2, 12, 12) \
    X3(2, 257, 2, 13, 13) \
    X3(2, 258, 2, 14, 14) \
    X3(2, 259, 2, 15, 15) \
    X3(2, 260, 3, 3, 12) \
    X3(2, 261, 3, 3, 14) \
    X3(2, 262, 3, 4, 5) \
    X3(2, 263, 3, 6, 7) \
    X3(2, 264, 3, 7, 8) \
    X3(2, 265, 3, 9, 10) \
    X3(2, 266, 3, 10, 11) \
    X3(2, 267, 3, 12, 13) \
    X3(2, 268, 3, 13, 14) \
    X3(2, 269, 3, 14, 15) \
    X3(2, 270, 4, 4, 12) \
    X3(2, 271, 4, 5, 13) \
    X3(2, 272, 4, 5, 15) \
    X3(2, 273, 4, 6, 10) \
    X3(2, 274, 4, 7, 9) \
    X3(2, 275, 4, 7, 11) \
    X3(2, 276, 5, 5, 12) \
    X3(2, 277, 5, 5, 14) \
    X3(2, 278, 5, 6, 11) \
    X3(2, 279, 5, 7, 10) \
    X3(2, 280, 5, 8, 9) \
    X3(2, 281, 5, 8, 11) \
    X3(2, 282, 6, 6, 12) \
    X3(2, 283, 6, 7, 13) \
    X3(2, 284, 6, 8, 14) \
    X3(2, 285, 7, 7, 12) \
    X3(2, 286, 7, 7, 14) \
    X3(2, 287, 7, 8, 13) \
    X3(2, 288, 7, 8, 15) \
    X3(2, 289, 8, 8, 12) \
    X3(2, 290, 9, 9, 12) \
    X3(2, 291, 9, 10, 13) \
    X3(2, 292, 9, 11, 14) \
    X3(2, 293, 10, 10, 12) \
    X3(2, 294, 10, 11, 13) \
    X3(2, 295, 10, 11, 15) \
    X3(2, 296, 11, 11, 12) \
    X3(2, 297, 11, 11, 14) \
    X3(2, 298, 12, 12, 12) \
    X3(2, 299, 12, 13, 13) \
    X3(2, 300, 12, 14, 14) \
    X3(2, 301, 12, 15, 15) \
    X3(2, 302, 13, 13, 14) \
    X3(2, 303, 13, 14, 15) \
    X3(3, 318, 0, 0, 3) \
    X3(3, 319, 0, 1, 4) \
    X3(3, 320, 0, 2, 7) \
    X3(3, 321, 0, 3, 6) \
    X3(3, 322, 0, 3, 8) \
    X3(3, 323, 0, 4, 9) \
    X3(3, 324, 0, 4, 11) \
    X3(3, 325, 0, 5, 10) \
    X3(3, 326, 0, 6, 13) \
    X3(3, 327, 0, 7, 12) \
    X3(3, 328, 0, 7, 14) \
    X3(3, 329, 0, 8, 13) \
    X3(3, 330, 0, 8, 15) \
    X3(3, 331, 1, 1, 3) \
    X3(3, 332, 1, 1, 13) \
    X3(3, 333, 1, 1, 15) \
    X3(3, 334, 1, 2, 10) \
    X3(3, 335, 1, 3, 9) \
    X3(3, 336, 1, 3, 11) \
    X3(3, 337, 1, 4, 6) \
    X3(3, 338, 1, 4, 8) \
    X3(3, 339, 1, 5, 7) \
    X3(3, 340, 1, 9, 13) \
    X3(3, 341, 1, 9, 15) \
    X3(3, 342, 1, 10, 12) \
    X3(3, 343, 1, 10, 14) \
    X3(3, 344, 1, 11, 13) \
    X3(3, 345, 1, 11, 15) \
    X3(3, 346, 2, 2, 3) \
    X3(3, 347, 2, 2, 13) \
    X3(3, 348, 2, 3, 12) \
    X3(3, 349, 2, 3, 14) \
    X3(3, 350, 2, 4, 5) \
    X3(3, 351, 2, 6, 7) \
    X3(3, 352, 2, 7, 8) \
    X3(3, 353, 2, 9, 10) \
    X3(3, 354, 2, 10, 11) \
    X3(3, 355, 2, 12, 13) \
    X3(3, 356, 2, 13, 14) \
    X3(3, 357, 2, 14, 15) \
    X3(3, 358, 3, 3, 3) \
    X3(3, 359, 3, 3, 13) \
    X3(3, 360, 3, 3, 15) \
    X3(3, 361, 3, 4, 4) \
    X3(3, 362, 3, 5, 5) \
    X3(3, 363, 3, 6, 6) \
    X3(3, 364, 3, 6, 8) \
    X3(3, 365, 3, 7, 7) \
    X3(3, 366, 3, 8, 8) \
    X3(3, 367, 3, 9, 9) \
    X3(3, 368, 3, 9, 11) \
    X3(3, 369, 3, 10, 10) \
    X3(3, 370, 3, 11, 11) \
    X3(3, 371, 3, 12, 12) \
    X3(3, 372, 3, 12, 14) \
    X3(3, 373, 3, 13, 13) \
    X3(3, 374, 3, 13, 15) \
    X3(3, 375, 3, 14, 14) \
    X3(3, 376, 3, 15, 15) \
    X3(3, 377, 4, 4, 13) \
    X3(3, 378, 4, 4, 15) \
    X3(3, 379, 4, 5, 12) \
    X3(3, 380, 4, 5, 14) \
    X3(3, 381, 4, 6, 9) \
    X3(3, 382, 4, 6, 11) \
    X3(3, 383, 4, 7, 10) \
    X3(3, 384, 4, 8, 9) \
    X3(3, 385, 4, 8, 11) \
    X3(3, 386, 5, 5, 13) \
    X3(3, 387, 5, 5, 15) \
    X3(3, 388, 5, 6, 10) \
    X3(3, 389, 5, 7, 9) \
    X3(3, 390, 5, 7, 11) \
    X3(3, 391, 5, 8, 10) \
    X3(3, 392, 6, 6, 13) \
    X3(3, 393, 6, 7, 12) \
    X3(3, 394, 6, 7, 14) \
    X3(3, 395, 6, 8, 13) \
    X3(3, 396, 6, 8, 15) \
    X3(3, 397, 7, 7, 13) \
    X3(3, 398, 7, 7, 15) \
    X3(3, 399, 7, 8, 12) \
    X3(3, 400, 7, 8, 14) \
    X3(3, 401, 8, 8, 13) \
    X3(3, 402, 8, 8, 15) \
    X3(3, 403, 9, 9, 13) \
    X3(3, 404, 9, 10, 12) \
    X3(3, 405, 9, 10, 14) \
    X3(3, 406, 9, 11, 13) \
    X3(3, 407, 9, 11, 15) \
    X3(3, 408, 10, 10, 13) \
    X3(3, 409, 10, 10, 15) \
    X3(3, 410, 10, 11, 12) \
    X3(3, 411, 10, 11, 14) \
    X3(3, 412, 11, 11, 13) \
    X3(3, 413, 11, 11, 15) \
    X3(3, 414, 12, 12, 13) \
    X3(3, 415, 12, 13, 14) \
    X3(3, 416, 12, 14, 15) \
    X3(3, 417, 13, 13, 13) \
    X3(3, 418, 13, 13, 15) \
    X3(3, 419, 13, 14, 14) \
    X3(3, 420, 13, 15, 15) \
    X3(3, 421, 14, 14, 15)
#define SXB_S1_M1_NUM_TERMS 94
#define SXB_S1_M1_TERMS(X1, X2, X3) \
    X1(0, 0, 0) \
    X2(0, 1, 0, 0) \
    X2(0, 2, 1, 1) \
    X2(0, 3, 2, 2) \
    X2(0, 4, 3, 3) \
    X2(0, 5, 4, 4) \
    X2(0, 6, 5, 5) \
    X2(0, 7, 6, 6) \
    X2(0, 8, 7, 7) \
    X2(0, 9, 8, 8) \
    X2(0, 10, 9, 9) \
    X2(0, 11, 10, 10) \
    X2(0, 12, 11, 11) \
    X2(0, 13, 12, 12) \
    X2(0, 14, 13, 13) \
    X2(0, 15, 14, 14) \
    X2(0, 16, 15, 15) \
    X3(0, 17, 0, 0, 0) \
    X3(0, 18, 0, 1, 1) \
    X3(0, 19, 0, 2, 2) \
    X3(0, 20, 0, 3, 3) \
    X3(0, 21, 0, 4, 4) \
    X3(0, 22, 0, 5, 5) \
    X3(0, 23, 0, 6, 6) \
    X3(0, 24, 0, 7, 7) \
    X3(0, 25, 0, 8, 8) \
    X3(0, 26, 0, 9, 9) \
    X3(0, 27, 0, 10, 10) \
    X3(0, 28, 0, 11, 11) \
    X3(0, 29, 0, 12, 12) \
    X3(0, 30, 0, 13, 13) \
    X3(0, 31, 0, 14, 14) \
    X3(0, 32, 0, 15, 15) \
    X3(0, 33, 1, 1, 6) \
    X3(0, 34, 1, 1, 8) \
    X3(0, 35, 1, 2, 5) \
    X3(0, 36, 1, 3, 4) \
    X3(0, 37, 1, 4, 13) \
    X3(0, 38, 1, 4, 15) \
    X3(0, 39, 1, 5, 12) \
    X3(0, 40, 1, 5, 14) \
    X3(0, 41, 1, 6, 11) \
    X3(0, 42, 1, 7, 10) \
    X3(0, 43, 1, 8, 9) \
    X3(0, 44, 1, 8, 11) \
    X3(0, 45, 2, 2, 6) \
    X3(0, 46, 2, 3, 7) \
    X3(0, 47, 2, 4, 10) \
    X3(0, 48, 2, 5, 11) \
    X3(0, 49, 2, 6, 12) \
    X3(0, 50, 2, 7, 13) \
    X3(0, 51, 2, 8, 14) \
    X3(0, 52, 3, 3, 6) \
    X3(0, 53, 3, 3, 8) \
    X3(0, 54, 3, 4, 9) \
    X3(0, 55, 3, 4, 11) \
    X3(0, 56, 3, 5, 10) \
    X3(0, 57, 3, 6, 13) \
    X3(0, 58, 3, 7, 12) \
    X3(0, 59, 3, 7, 14) \
    X3(0, 60, 3, 8, 13) \
    X3(0, 61, 3, 8, 15) \
    X3(0, 62, 4, 4, 6) \
    X3(0, 63, 4, 5, 7) \
    X3(0, 64, 4, 9, 13) \
    X3(0, 65, 4, 10, 12) \
    X3(0, 66, 4, 11, 13) \
    X3(0, 67, 4, 11, 15) \
    X3(0, 68, 5, 5, 6) \
    X3(0, 69, 5, 5, 8) \
    X3(0, 70, 5, 9, 14) \
    X3(0, 71, 5, 10, 13) \
    X3(0, 72, 5, 10, 15) \
    X3(0, 73, 5, 11, 12) \
    X3(0, 74, 5, 11, 14) \
    X3(0, 75, 6, 6, 6) \
    X3(0, 76, 6, 7, 7) \
    X3(0, 77, 6, 8, 8) \
    X3(0, 78, 6, 9, 9) \
    X3(0, 79, 6, 11, 11) \
    X3(0, 80, 6, 12, 12) \
    X3(0, 81, 6, 13, 13) \
    X3(0, 82, 6, 15, 15) \
    X3(0, 83, 7, 7, 8) \
    X3(0, 84, 7, 9, 10) \
    X3(0, 85, 7, 10, 11) \
    X3(0, 86, 7, 12, 13) \
    X3(0, 87, 7, 13, 14) \
    X3(0, 88, 7, 14, 15) \
    X3(0, 89, 8, 9, 11) \
    X3(0, 90, 8, 11, 11) \
    X3(0, 91, 8, 12, 14) \
    X3(0, 92, 8, 13, 13) \
    X3(0, 93, 8, 13, 15)
#define SXB_S1_M0_FORWARD_BODY \
      o[0] = f2_fma(W(0), x[0], o[0]); \
      o[1] = f2_fma(W(94), x[1], o[1]); \
      o[2] = f2_fma(W(212), x[2], o[2]); \
      o[3] = f2_fma(W(304), x[3], o[3]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); o[0] = f2_fma(p, f2_fma(W(17), x[0], W(1)), o[0]); o[1] = f2_fma(p, f2_mul(W(108), x[1]), o[1]); o[2] = f2_fma(p, f2_mul(W(222), x[2]), o[2]); o[3] = f2_fma(p, f2_mul(W(318), x[3]), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); o[0] = f2_fma(p, f2_mul(W(18), x[1]), o[0]); o[1] = f2_fma(p, f2_fma(W(110), x[8], f2_fma(W(109), x[6], W(95))), o[1]); o[2] = f2_fma(p, f2_mul(W(223), x[5]), o[2]); o[3] = f2_fma(p, f2_mul(W(319), x[4]), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); o[0] = f2_fma(p, f2_mul(W(19), x[2]), o[0]); o[1] = f2_fma(p, f2_mul(W(111), x[5]), o[1]); o[2] = f2_fma(p, f2_fma(W(224), x[6], W(213)), o[2]); o[3] = f2_fma(p, f2_mul(W(320), x[7]), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); o[0] = f2_fma(p, f2_mul(W(20), x[3]), o[0]); o[1] = f2_fma(p, f2_mul(W(112), x[4]), o[1]); o[2] = f2_fma(p, f2_mul(W(225), x[7]), o[2]); o[3] = f2_fma(p, f2_fma(W(322), x[8], f2_fma(W(321), x[6], W(305))), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); o[0] = f2_fma(p, f2_mul(W(21), x[4]), o[0]); o[1] = f2_fma(p, f2_fma(W(114), x[15], f2_mul(W(113), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(226), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(324), x[11], f2_mul(W(323), x[9])), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); o[0] = f2_fma(p, f2_mul(W(22), x[5]), o[0]); o[1] = f2_fma(p, f2_fma(W(116), x[14], f2_mul(W(115), x[12])), o[1]); o[2] = f2_fma(p, f2_mul(W(227), x[11]), o[2]); o[3] = f2_fma(p, f2_mul(W(325), x[10]), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); o[0] = f2_fma(p, f2_mul(W(23), x[6]), o[0]); o[1] = f2_fma(p, f2_mul(W(117), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(228), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(326), x[13]), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); o[0] = f2_fma(p, f2_mul(W(24), x[7]), o[0]); o[1] = f2_fma(p, f2_mul(W(118), x[10]), o[1]); o[2] = f2_fma(p, f2_mul(W(229), x[13]), o[2]); o[3] = f2_fma(p, f2_fma(W(328), x[14], f2_mul(W(327), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); o[0] = f2_fma(p, f2_mul(W(25), x[8]), o[0]); o[1] = f2_fma(p, f2_fma(W(120), x[11], f2_mul(W(119), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(230), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(330), x[15], f2_mul(W(329), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); o[0] = f2_fma(p, f2_mul(W(26), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); o[0] = f2_fma(p, f2_mul(W(27), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); o[0] = f2_fma(p, f2_mul(W(28), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); o[0] = f2_fma(p, f2_mul(W(29), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); o[0] = f2_fma(p, f2_mul(W(30), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); o[0] = f2_fma(p, f2_mul(W(31), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); o[0] = f2_fma(p, f2_mul(W(32), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); o[0] = f2_fma(p, f2_fma(W(34), x[8], f2_fma(W(33), x[6], W(2))), o[0]); o[1] = f2_fma(p, f2_fma(W(123), x[11], f2_fma(W(122), x[9], f2_mul(W(121), x[1]))), o[1]); o[2] = f2_fma(p, f2_fma(W(233), x[14], f2_fma(W(232), x[12], f2_mul(W(231), x[2]))), o[2]); o[3] = f2_fma(p, f2_fma(W(333), x[15], f2_fma(W(332), x[13], f2_mul(W(331), x[3]))), o[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); o[0] = f2_fma(p, f2_mul(W(35), x[5]), o[0]); o[1] = f2_fma(p, f2_fma(W(126), x[14], f2_fma(W(125), x[12], f2_mul(W(124), x[2]))), o[1]); o[2] = f2_fma(p, f2_mul(W(234), x[11]), o[2]); o[3] = f2_fma(p, f2_mul(W(334), x[10]), o[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); o[0] = f2_fma(p, f2_mul(W(36), x[4]), o[0]); o[1] = f2_fma(p, f2_fma(W(129), x[15], f2_fma(W(128), x[13], f2_mul(W(127), x[3]))), o[1]); o[2] = f2_fma(p, f2_mul(W(235), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(336), x[11], f2_mul(W(335), x[9])), o[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); o[0] = f2_fma(p, f2_fma(W(38), x[15], f2_mul(W(37), x[13])), o[0]); o[1] = f2_fma(p, f2_mul(W(130), x[4]), o[1]); o[2] = f2_fma(p, f2_mul(W(236), x[7]), o[2]); o[3] = f2_fma(p, f2_fma(W(338), x[8], f2_fma(W(337), x[6], W(306))), o[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); o[0] = f2_fma(p, f2_fma(W(40), x[14], f2_mul(W(39), x[12])), o[0]); o[1] = f2_fma(p, f2_mul(W(131), x[5]), o[1]); o[2] = f2_fma(p, f2_fma(W(238), x[8], f2_fma(W(237), x[6], W(214))), o[2]); o[3] = f2_fma(p, f2_mul(W(339), x[7]), o[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); o[0] = f2_fma(p, f2_mul(W(41), x[11]), o[0]); o[1] = f2_fma(p, f2_fma(W(133), x[8], f2_fma(W(132), x[6], W(96))), o[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); o[0] = f2_fma(p, f2_mul(W(42), x[10]), o[0]); o[1] = f2_fma(p, f2_mul(W(134), x[7]), o[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); o[0] = f2_fma(p, f2_fma(W(44), x[11], f2_mul(W(43), x[9])), o[0]); o[1] = f2_fma(p, f2_fma(W(135), x[8], W(97)), o[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[9]); o[1] = f2_fma(p, f2_fma(W(137), x[11], f2_mul(W(136), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(239), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(341), x[15], f2_mul(W(340), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[10]); o[1] = f2_fma(p, f2_mul(W(138), x[10]), o[1]); o[2] = f2_fma(p, f2_fma(W(241), x[15], f2_mul(W(240), x[13])), o[2]); o[3] = f2_fma(p, f2_fma(W(343), x[14], f2_mul(W(342), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[11]); o[1] = f2_fma(p, f2_mul(W(139), x[11]), o[1]); o[2] = f2_fma(p, f2_fma(W(243), x[14], f2_mul(W(242), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(345), x[15], f2_mul(W(344), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[12]); o[1] = f2_fma(p, f2_fma(W(141), x[14], f2_mul(W(140), x[12])), o[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[13]); o[1] = f2_fma(p, f2_fma(W(143), x[15], f2_mul(W(142), x[13])), o[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[14]); o[1] = f2_fma(p, f2_mul(W(144), x[14]), o[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[15]); o[1] = f2_fma(p, f2_mul(W(145), x[15]), o[1]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); o[0] = f2_fma(p, f2_fma(W(45), x[6], W(3)), o[0]); o[1] = f2_fma(p, f2_mul(W(146), x[11]), o[1]); o[2] = f2_fma(p, f2_fma(W(245), x[12], f2_mul(W(244), x[2])), o[2]); o[3] = f2_fma(p, f2_fma(W(347), x[13], f2_mul(W(346), x[3])), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); o[0] = f2_fma(p, f2_mul(W(46), x[7]), o[0]); o[1] = f2_fma(p, f2_mul(W(147), x[10]), o[1]); o[2] = f2_fma(p, f2_fma(W(247), x[13], f2_mul(W(246), x[3])), o[2]); o[3] = f2_fma(p, f2_fma(W(349), x[14], f2_mul(W(348), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); o[0] = f2_fma(p, f2_mul(W(47), x[10]), o[0]); o[1] = f2_fma(p, f2_mul(W(148), x[7]), o[1]); o[2] = f2_fma(p, f2_mul(W(248), x[4]), o[2]); o[3] = f2_fma(p, f2_mul(W(350), x[5]), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); o[0] = f2_fma(p, f2_mul(W(48), x[11]), o[0]); o[1] = f2_fma(p, f2_fma(W(150), x[8], f2_fma(W(149), x[6], W(98))), o[1]); o[2] = f2_fma(p, f2_mul(W(249), x[5]), o[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); o[0] = f2_fma(p, f2_mul(W(49), x[12]), o[0]); o[2] = f2_fma(p, f2_fma(W(250), x[6], W(215)), o[2]); o[3] = f2_fma(p, f2_mul(W(351), x[7]), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); o[0] = f2_fma(p, f2_mul(W(50), x[13]), o[0]); o[2] = f2_fma(p, f2_mul(W(251), x[7]), o[2]); o[3] = f2_fma(p, f2_fma(W(352), x[8], W(307)), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); o[0] = f2_fma(p, f2_mul(W(51), x[14]), o[0]); o[2] = f2_fma(p, f2_mul(W(252), x[8]), o[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[9]); o[1] = f2_fma(p, f2_mul(W(151), x[14]), o[1]); o[2] = f2_fma(p, f2_mul(W(253), x[9]), o[2]); o[3] = f2_fma(p, f2_mul(W(353), x[10]), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[10]); o[1] = f2_fma(p, f2_fma(W(153), x[15], f2_mul(W(152), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(254), x[10]), o[2]); o[3] = f2_fma(p, f2_mul(W(354), x[11]), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[11]); o[1] = f2_fma(p, f2_fma(W(155), x[14], f2_mul(W(154), x[12])), o[1]); o[2] = f2_fma(p, f2_mul(W(255), x[11]), o[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[12]); o[2] = f2_fma(p, f2_mul(W(256), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(355), x[13]), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[13]); o[2] = f2_fma(p, f2_mul(W(257), x[13]), o[2]); o[3] = f2_fma(p, f2_mul(W(356), x[14]), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[14]); o[2] = f2_fma(p, f2_mul(W(258), x[14]), o[2]); o[3] = f2_fma(p, f2_mul(W(357), x[15]), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[15]); o[2] = f2_fma(p, f2_mul(W(259), x[15]), o[2]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); o[0] = f2_fma(p, f2_fma(W(53), x[8], f2_fma(W(52), x[6], W(4))), o[0]); o[1] = f2_fma(p, f2_fma(W(157), x[11], f2_mul(W(156), x[9])), o[1]); o[2] = f2_fma(p, f2_fma(W(261), x[14], f2_mul(W(260), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(360), x[15], f2_fma(W(359), x[13], f2_mul(W(358), x[3]))), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); o[0] = f2_fma(p, f2_fma(W(55), x[11], f2_mul(W(54), x[9])), o[0]); o[1] = f2_fma(p, f2_fma(W(159), x[8], f2_fma(W(158), x[6], W(99))), o[1]); o[2] = f2_fma(p, f2_mul(W(262), x[5]), o[2]); o[3] = f2_fma(p, f2_mul(W(361), x[4]), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); o[0] = f2_fma(p, f2_mul(W(56), x[10]), o[0]); o[1] = f2_fma(p, f2_mul(W(160), x[7]), o[1]); o[3] = f2_fma(p, f2_mul(W(362), x[5]), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); o[0] = f2_fma(p, f2_mul(W(57), x[13]), o[0]); o[2] = f2_fma(p, f2_mul(W(263), x[7]), o[2]); o[3] = f2_fma(p, f2_fma(W(364), x[8], f2_fma(W(363), x[6], W(308))), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); o[0] = f2_fma(p, f2_fma(W(59), x[14], f2_mul(W(58), x[12])), o[0]); o[2] = f2_fma(p, f2_fma(W(264), x[8], W(216)), o[2]); o[3] = f2_fma(p, f2_mul(W(365), x[7]), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); o[0] = f2_fma(p, f2_fma(W(61), x[15], f2_mul(W(60), x[13])), o[0]); o[3] = f2_fma(p, f2_fma(W(366), x[8], W(309)), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[9]); o[1] = f2_fma(p, f2_fma(W(162), x[15], f2_mul(W(161), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(265), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(368), x[11], f2_mul(W(367), x[9])), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[10]); o[1] = f2_fma(p, f2_fma(W(164), x[14], f2_mul(W(163), x[12])), o[1]); o[2] = f2_fma(p, f2_mul(W(266), x[11]), o[2]); o[3] = f2_fma(p, f2_mul(W(369), x[10]), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[11]); o[1] = f2_fma(p, f2_fma(W(166), x[15], f2_mul(W(165), x[13])), o[1]); o[3] = f2_fma(p, f2_mul(W(370), x[11]), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[12]); o[2] = f2_fma(p, f2_mul(W(267), x[13]), o[2]); o[3] = f2_fma(p, f2_fma(W(372), x[14], f2_mul(W(371), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[13]); o[2] = f2_fma(p, f2_mul(W(268), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(374), x[15], f2_mul(W(373), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[14]); o[2] = f2_fma(p, f2_mul(W(269), x[15]), o[2]); o[3] = f2_fma(p, f2_mul(W(375), x[14]), o[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[15]); o[3] = f2_fma(p, f2_mul(W(376), x[15]), o[3]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); o[0] = f2_fma(p, f2_fma(W(62), x[6], W(5)), o[0]); o[1] = f2_fma(p, f2_fma(W(168), x[11], f2_mul(W(167), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(270), x[12]), o[2]); o[3] = f2_fma(p, f2_fma(W(378), x[15], f2_mul(W(377), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); o[0] = f2_fma(p, f2_mul(W(63), x[7]), o[0]); o[1] = f2_fma(p, f2_mul(W(169), x[10]), o[1]); o[2] = f2_fma(p, f2_fma(W(272), x[15], f2_mul(W(271), x[13])), o[2]); o[3] = f2_fma(p, f2_fma(W(380), x[14], f2_mul(W(379), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[4], x[6]); o[1] = f2_fma(p, f2_fma(W(171), x[15], f2_mul(W(170), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(273), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(382), x[11], f2_mul(W(381), x[9])), o[3]); } \
      { const unsigned long long p = f2_mul(x[4], x[7]); o[1] = f2_fma(p, f2_fma(W(173), x[14], f2_mul(W(172), x[12])), o[1]); o[2] = f2_fma(p, f2_fma(W(275), x[11], f2_mul(W(274), x[9])), o[2]); o[3] = f2_fma(p, f2_mul(W(383), x[10]), o[3]); } \
      { const unsigned long long p = f2_mul(x[4], x[8]); o[1] = f2_fma(p, f2_fma(W(175), x[15], f2_mul(W(174), x[13])), o[1]); o[3] = f2_fma(p, f2_fma(W(385), x[11], f2_mul(W(384), x[9])), o[3]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); o[0] = f2_fma(p, f2_mul(W(64), x[13]), o[0]); o[3] = f2_fma(p, W(310), o[3]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); o[0] = f2_fma(p, f2_mul(W(65), x[12]), o[0]); o[2] = f2_fma(p, W(217), o[2]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); o[0] = f2_fma(p, f2_fma(W(67), x[15], f2_mul(W(66), x[13])), o[0]); o[3] = f2_fma(p, W(311), o[3]); } \
      { const unsigned long long p = f2_mul(x[4], x[13]); o[1] = f2_fma(p, W(100), o[1]); } \
      { const unsigned long long p = f2_mul(x[4], x[15]); o[1] = f2_fma(p, W(101), o[1]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); o[0] = f2_fma(p, f2_fma(W(69), x[8], f2_fma(W(68), x[6], W(6))), o[0]); o[1] = f2_fma(p, f2_fma(W(177), x[11], f2_mul(W(176), x[9])), o[1]); o[2] = f2_fma(p, f2_fma(W(277), x[14], f2_mul(W(276), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(387), x[15], f2_mul(W(386), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[5], x[6]); o[1] = f2_fma(p, f2_fma(W(179), x[14], f2_mul(W(178), x[12])), o[1]); o[2] = f2_fma(p, f2_mul(W(278), x[11]), o[2]); o[3] = f2_fma(p, f2_mul(W(388), x[10]), o[3]); } \
      { const unsigned long long p = f2_mul(x[5], x[7]); o[1] = f2_fma(p, f2_fma(W(181), x[15], f2_mul(W(180), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(279), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(390), x[11], f2_mul(W(389), x[9])), o[3]); } \
      { const unsigned long long p = f2_mul(x[5], x[8]); o[1] = f2_fma(p, f2_fma(W(183), x[14], f2_mul(W(182), x[12])), o[1]); o[2] = f2_fma(p, f2_fma(W(281), x[11], f2_mul(W(280), x[9])), o[2]); o[3] = f2_fma(p, f2_mul(W(391), x[10]), o[3]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); o[0] = f2_fma(p, f2_mul(W(70), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); o[0] = f2_fma(p, f2_fma(W(72), x[15], f2_mul(W(71), x[13])), o[0]); o[3] = f2_fma(p, W(312), o[3]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); o[0] = f2_fma(p, f2_fma(W(74), x[14], f2_mul(W(73), x[12])), o[0]); o[2] = f2_fma(p, W(218), o[2]); } \
      { const unsigned long long p = f2_mul(x[5], x[12]); o[1] = f2_fma(p, W(102), o[1]); } \
      { const unsigned long long p = f2_mul(x[5], x[14]); o[1] = f2_fma(p, W(103), o[1]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); o[0] = f2_fma(p, f2_fma(W(75), x[6], W(7)), o[0]); o[1] = f2_fma(p, f2_mul(W(184), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(282), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(392), x[13]), o[3]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); o[0] = f2_fma(p, f2_mul(W(76), x[7]), o[0]); o[1] = f2_fma(p, f2_mul(W(185), x[10]), o[1]); o[2] = f2_fma(p, f2_mul(W(283), x[13]), o[2]); o[3] = f2_fma(p, f2_fma(W(394), x[14], f2_mul(W(393), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); o[0] = f2_fma(p, f2_mul(W(77), x[8]), o[0]); o[1] = f2_fma(p, f2_fma(W(187), x[11], f2_mul(W(186), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(284), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(396), x[15], f2_mul(W(395), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); o[0] = f2_fma(p, f2_mul(W(78), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); o[0] = f2_fma(p, f2_mul(W(79), x[11]), o[0]); o[1] = f2_fma(p, W(104), o[1]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); o[0] = f2_fma(p, f2_mul(W(80), x[12]), o[0]); o[2] = f2_fma(p, W(219), o[2]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); o[0] = f2_fma(p, f2_mul(W(81), x[13]), o[0]); o[3] = f2_fma(p, W(313), o[3]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); o[0] = f2_fma(p, f2_mul(W(82), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); o[0] = f2_fma(p, f2_fma(W(83), x[8], W(8)), o[0]); o[1] = f2_fma(p, f2_fma(W(189), x[11], f2_mul(W(188), x[9])), o[1]); o[2] = f2_fma(p, f2_fma(W(286), x[14], f2_mul(W(285), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(398), x[15], f2_mul(W(397), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[7], x[8]); o[1] = f2_fma(p, f2_mul(W(190), x[10]), o[1]); o[2] = f2_fma(p, f2_fma(W(288), x[15], f2_mul(W(287), x[13])), o[2]); o[3] = f2_fma(p, f2_fma(W(400), x[14], f2_mul(W(399), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); o[0] = f2_fma(p, f2_mul(W(84), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); o[0] = f2_fma(p, f2_mul(W(85), x[11]), o[0]); o[1] = f2_fma(p, W(105), o[1]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); o[0] = f2_fma(p, f2_mul(W(86), x[13]), o[0]); o[3] = f2_fma(p, W(314), o[3]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); o[0] = f2_fma(p, f2_mul(W(87), x[14]), o[0]); o[2] = f2_fma(p, W(220), o[2]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); o[0] = f2_fma(p, f2_mul(W(88), x[15]), o[0]); o[3] = f2_fma(p, W(315), o[3]); } \
      { const unsigned long long p = f2_mul(x[8], x[8]); o[0] = f2_fma(p, W(9), o[0]); o[1] = f2_fma(p, f2_fma(W(192), x[11], f2_mul(W(191), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(289), x[12]), o[2]); o[3] = f2_fma(p, f2_fma(W(402), x[15], f2_mul(W(401), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); o[0] = f2_fma(p, f2_mul(W(89), x[11]), o[0]); o[1] = f2_fma(p, W(106), o[1]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); o[0] = f2_fma(p, f2_mul(W(90), x[11]), o[0]); o[1] = f2_fma(p, W(107), o[1]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); o[0] = f2_fma(p, f2_mul(W(91), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); o[0] = f2_fma(p, f2_fma(W(93), x[15], f2_mul(W(92), x[13])), o[0]); o[3] = f2_fma(p, W(316), o[3]); } \
      { const unsigned long long p = f2_mul(x[8], x[14]); o[2] = f2_fma(p, W(221), o[2]); } \
      { const unsigned long long p = f2_mul(x[8], x[15]); o[3] = f2_fma(p, W(317), o[3]); } \
      { const unsigned long long p = f2_mul(x[9], x[9]); o[0] = f2_fma(p, W(10), o[0]); o[1] = f2_fma(p, f2_mul(W(193), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(290), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(403), x[13]), o[3]); } \
      { const unsigned long long p = f2_mul(x[9], x[10]); o[1] = f2_fma(p, f2_mul(W(194), x[10]), o[1]); o[2] = f2_fma(p, f2_mul(W(291), x[13]), o[2]); o[3] = f2_fma(p, f2_fma(W(405), x[14], f2_mul(W(404), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[9], x[11]); o[1] = f2_fma(p, f2_mul(W(195), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(292), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(407), x[15], f2_mul(W(406), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[9], x[12]); o[1] = f2_fma(p, f2_mul(W(196), x[14]), o[1]); } \
      { const unsigned long long p = f2_mul(x[9], x[13]); o[1] = f2_fma(p, f2_fma(W(198), x[15], f2_mul(W(197), x[13])), o[1]); } \
      { const unsigned long long p = f2_mul(x[9], x[14]); o[1] = f2_fma(p, f2_mul(W(199), x[14]), o[1]); } \
      { const unsigned long long p = f2_mul(x[10], x[10]); o[0] = f2_fma(p, W(11), o[0]); o[1] = f2_fma(p, f2_mul(W(200), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(293), x[12]), o[2]); o[3] = f2_fma(p, f2_fma(W(409), x[15], f2_mul(W(408), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[10], x[11]); o[2] = f2_fma(p, f2_fma(W(295), x[15], f2_mul(W(294), x[13])), o[2]); o[3] = f2_fma(p, f2_fma(W(411), x[14], f2_mul(W(410), x[12])), o[3]); } \
      { const unsigned long long p = f2_mul(x[10], x[12]); o[1] = f2_fma(p, f2_fma(W(202), x[15], f2_mul(W(201), x[13])), o[1]); } \
      { const unsigned long long p = f2_mul(x[10], x[13]); o[1] = f2_fma(p, f2_mul(W(203), x[14]), o[1]); } \
      { const unsigned long long p = f2_mul(x[10], x[14]); o[1] = f2_fma(p, f2_mul(W(204), x[15]), o[1]); } \
      { const unsigned long long p = f2_mul(x[11], x[11]); o[0] = f2_fma(p, W(12), o[0]); o[1] = f2_fma(p, f2_mul(W(205), x[11]), o[1]); o[2] = f2_fma(p, f2_fma(W(297), x[14], f2_mul(W(296), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(413), x[15], f2_mul(W(412), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[11], x[12]); o[1] = f2_fma(p, f2_fma(W(207), x[14], f2_mul(W(206), x[12])), o[1]); } \
      { const unsigned long long p = f2_mul(x[11], x[13]); o[1] = f2_fma(p, f2_fma(W(209), x[15], f2_mul(W(208), x[13])), o[1]); } \
      { const unsigned long long p = f2_mul(x[11], x[14]); o[1] = f2_fma(p, f2_mul(W(210), x[14]), o[1]); } \
      { const unsigned long long p = f2_mul(x[11], x[15]); o[1] = f2_fma(p, f2_mul(W(211), x[15]), o[1]); } \
      { const unsigned long long p = f2_mul(x[12], x[12]); o[0] = f2_fma(p, W(13), o[0]); o[2] = f2_fma(p, f2_mul(W(298), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(414), x[13]), o[3]); } \
      { const unsigned long long p = f2_mul(x[12], x[13]); o[2] = f2_fma(p, f2_mul(W(299), x[13]), o[2]); o[3] = f2_fma(p, f2_mul(W(415), x[14]), o[3]); } \
      { const unsigned long long p = f2_mul(x[12], x[14]); o[2] = f2_fma(p, f2_mul(W(300), x[14]), o[2]); o[3] = f2_fma(p, f2_mul(W(416), x[15]), o[3]); } \
      { const unsigned long long p = f2_mul(x[12], x[15]); o[2] = f2_fma(p, f2_mul(W(301), x[15]), o[2]); } \
      { const unsigned long long p = f2_mul(x[13], x[13]); o[0] = f2_fma(p, W(14), o[0]); o[2] = f2_fma(p, f2_mul(W(302), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(418), x[15], f2_mul(W(417), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[13], x[14]); o[2] = f2_fma(p, f2_mul(W(303), x[15]), o[2]); o[3] = f2_fma(p, f2_mul(W(419), x[14]), o[3]); } \
      { const unsigned long long p = f2_mul(x[13], x[15]); o[3] = f2_fma(p, f2_mul(W(420), x[15]), o[3]); } \
      { const unsigned long long p = f2_mul(x[14], x[14]); o[0] = f2_fma(p, W(15), o[0]); o[3] = f2_fma(p, f2_mul(W(421), x[15]), o[3]); } \
      { const unsigned long long p = f2_mul(x[15], x[15]); o[0] = f2_fma(p, W(16), o[0]); }
#define SXB_S1_M0_REVERSE_BODY \
      g[0] = f2_fma(W(0), adj[0], g[0]); \
      g[1] = f2_fma(W(94), adj[1], g[1]); \
      g[2] = f2_fma(W(212), adj[2], g[2]); \
      g[3] = f2_fma(W(304), adj[3], g[3]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); unsigned long long v; v = f2_mul(W(1), adj[0]); { const unsigned long long s = f2_mul(W(17), adj[0]); g[0] = f2_fma(s, p, g[0]); v = f2_fma(s, x[0], v); } { const unsigned long long s = f2_mul(W(108), adj[1]); g[1] = f2_fma(s, p, g[1]); v = f2_fma(s, x[1], v); } { const unsigned long long s = f2_mul(W(222), adj[2]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(318), adj[3]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } g[0] = f2_fma(v, x[0], g[0]); g[0] = f2_fma(v, x[0], g[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); unsigned long long v; v = f2_mul(W(95), adj[1]); { const unsigned long long s = f2_mul(W(18), adj[0]); g[1] = f2_fma(s, p, g[1]); v = f2_fma(s, x[1], v); } { const unsigned long long s = f2_mul(W(319), adj[3]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(223), adj[2]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(109), adj[1]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(110), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[0] = f2_fma(v, x[1], g[0]); g[1] = f2_fma(v, x[0], g[1]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); unsigned long long v; v = f2_mul(W(213), adj[2]); { const unsigned long long s = f2_mul(W(19), adj[0]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(111), adj[1]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(224), adj[2]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(320), adj[3]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } g[0] = f2_fma(v, x[2], g[0]); g[2] = f2_fma(v, x[0], g[2]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); unsigned long long v; v = f2_mul(W(305), adj[3]); { const unsigned long long s = f2_mul(W(20), adj[0]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(112), adj[1]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(321), adj[3]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(225), adj[2]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(322), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[0] = f2_fma(v, x[3], g[0]); g[3] = f2_fma(v, x[0], g[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(21), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } { const unsigned long long s = f2_mul(W(323), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(226), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(324), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(113), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(114), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[4], g[0]); g[4] = f2_fma(v, x[0], g[4]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(22), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } { const unsigned long long s = f2_mul(W(325), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(227), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(115), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(116), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[0] = f2_fma(v, x[5], g[0]); g[5] = f2_fma(v, x[0], g[5]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(23), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_mul(s, x[6]); } { const unsigned long long s = f2_mul(W(117), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(228), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(326), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[0] = f2_fma(v, x[6], g[0]); g[6] = f2_fma(v, x[0], g[6]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(24), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } { const unsigned long long s = f2_mul(W(118), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(327), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(229), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(328), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[0] = f2_fma(v, x[7], g[0]); g[7] = f2_fma(v, x[0], g[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(25), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } { const unsigned long long s = f2_mul(W(119), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(120), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(329), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(230), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(330), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[8], g[0]); g[8] = f2_fma(v, x[0], g[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(26), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[0] = f2_fma(v, x[9], g[0]); g[9] = f2_fma(v, x[0], g[9]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(27), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[0] = f2_fma(v, x[10], g[0]); g[10] = f2_fma(v, x[0], g[10]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(28), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[0] = f2_fma(v, x[11], g[0]); g[11] = f2_fma(v, x[0], g[11]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(29), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[0] = f2_fma(v, x[12], g[0]); g[12] = f2_fma(v, x[0], g[12]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(30), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[0] = f2_fma(v, x[13], g[0]); g[13] = f2_fma(v, x[0], g[13]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(31), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[0] = f2_fma(v, x[14], g[0]); g[14] = f2_fma(v, x[0], g[14]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(32), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[0] = f2_fma(v, x[15], g[0]); g[15] = f2_fma(v, x[0], g[15]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); unsigned long long v; v = f2_mul(W(2), adj[0]); { const unsigned long long s = f2_mul(W(121), adj[1]); g[1] = f2_fma(s, p, g[1]); v = f2_fma(s, x[1], v); } { const unsigned long long s = f2_mul(W(231), adj[2]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(331), adj[3]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(33), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(34), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(122), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(123), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(232), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(332), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(233), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(333), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[1], g[1]); g[1] = f2_fma(v, x[1], g[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(124), adj[1]); g[2] = f2_fma(s, p, g[2]); v = f2_mul(s, x[2]); } { const unsigned long long s = f2_mul(W(35), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(334), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(234), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(125), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(126), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[2], g[1]); g[2] = f2_fma(v, x[1], g[2]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(127), adj[1]); g[3] = f2_fma(s, p, g[3]); v = f2_mul(s, x[3]); } { const unsigned long long s = f2_mul(W(36), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(335), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(235), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(336), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(128), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(129), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[3], g[1]); g[3] = f2_fma(v, x[1], g[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); unsigned long long v; v = f2_mul(W(306), adj[3]); { const unsigned long long s = f2_mul(W(130), adj[1]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(337), adj[3]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(236), adj[2]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(338), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(37), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(38), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[4], g[1]); g[4] = f2_fma(v, x[1], g[4]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); unsigned long long v; v = f2_mul(W(214), adj[2]); { const unsigned long long s = f2_mul(W(131), adj[1]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(237), adj[2]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(339), adj[3]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(238), adj[2]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(39), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(40), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[5], g[1]); g[5] = f2_fma(v, x[1], g[5]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); unsigned long long v; v = f2_mul(W(96), adj[1]); { const unsigned long long s = f2_mul(W(132), adj[1]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(133), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(41), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[1] = f2_fma(v, x[6], g[1]); g[6] = f2_fma(v, x[1], g[6]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(134), adj[1]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } { const unsigned long long s = f2_mul(W(42), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } g[1] = f2_fma(v, x[7], g[1]); g[7] = f2_fma(v, x[1], g[7]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); unsigned long long v; v = f2_mul(W(97), adj[1]); { const unsigned long long s = f2_mul(W(135), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(43), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(44), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[1] = f2_fma(v, x[8], g[1]); g[8] = f2_fma(v, x[1], g[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(136), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(137), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(340), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(239), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(341), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[9], g[1]); g[9] = f2_fma(v, x[1], g[9]); } \
      { const unsigned long long p = f2_mul(x[1], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(138), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(342), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(240), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(343), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(241), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[10], g[1]); g[10] = f2_fma(v, x[1], g[10]); } \
      { const unsigned long long p = f2_mul(x[1], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(139), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } { const unsigned long long s = f2_mul(W(242), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(344), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(243), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(345), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[11], g[1]); g[11] = f2_fma(v, x[1], g[11]); } \
      { const unsigned long long p = f2_mul(x[1], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(140), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(141), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[12], g[1]); g[12] = f2_fma(v, x[1], g[12]); } \
      { const unsigned long long p = f2_mul(x[1], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(142), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(143), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[13], g[1]); g[13] = f2_fma(v, x[1], g[13]); } \
      { const unsigned long long p = f2_mul(x[1], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(144), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[1] = f2_fma(v, x[14], g[1]); g[14] = f2_fma(v, x[1], g[14]); } \
      { const unsigned long long p = f2_mul(x[1], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(145), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[1] = f2_fma(v, x[15], g[1]); g[15] = f2_fma(v, x[1], g[15]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); unsigned long long v; v = f2_mul(W(3), adj[0]); { const unsigned long long s = f2_mul(W(244), adj[2]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(346), adj[3]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(45), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(146), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(245), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(347), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[2] = f2_fma(v, x[2], g[2]); g[2] = f2_fma(v, x[2], g[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(246), adj[2]); g[3] = f2_fma(s, p, g[3]); v = f2_mul(s, x[3]); } { const unsigned long long s = f2_mul(W(46), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(147), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(348), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(247), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(349), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[3], g[2]); g[3] = f2_fma(v, x[2], g[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(248), adj[2]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } { const unsigned long long s = f2_mul(W(350), adj[3]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(148), adj[1]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(47), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } g[2] = f2_fma(v, x[4], g[2]); g[4] = f2_fma(v, x[2], g[4]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); unsigned long long v; v = f2_mul(W(98), adj[1]); { const unsigned long long s = f2_mul(W(249), adj[2]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(149), adj[1]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(150), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(48), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[2] = f2_fma(v, x[5], g[2]); g[5] = f2_fma(v, x[2], g[5]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); unsigned long long v; v = f2_mul(W(215), adj[2]); { const unsigned long long s = f2_mul(W(250), adj[2]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(351), adj[3]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(49), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } g[2] = f2_fma(v, x[6], g[2]); g[6] = f2_fma(v, x[2], g[6]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); unsigned long long v; v = f2_mul(W(307), adj[3]); { const unsigned long long s = f2_mul(W(251), adj[2]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(352), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(50), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[2] = f2_fma(v, x[7], g[2]); g[7] = f2_fma(v, x[2], g[7]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(252), adj[2]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } { const unsigned long long s = f2_mul(W(51), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[8], g[2]); g[8] = f2_fma(v, x[2], g[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(253), adj[2]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(353), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(151), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[9], g[2]); g[9] = f2_fma(v, x[2], g[9]); } \
      { const unsigned long long p = f2_mul(x[2], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(254), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(354), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(152), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(153), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[2] = f2_fma(v, x[10], g[2]); g[10] = f2_fma(v, x[2], g[10]); } \
      { const unsigned long long p = f2_mul(x[2], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(255), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } { const unsigned long long s = f2_mul(W(154), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(155), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[11], g[2]); g[11] = f2_fma(v, x[2], g[11]); } \
      { const unsigned long long p = f2_mul(x[2], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(256), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(355), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[2] = f2_fma(v, x[12], g[2]); g[12] = f2_fma(v, x[2], g[12]); } \
      { const unsigned long long p = f2_mul(x[2], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(257), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(356), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[13], g[2]); g[13] = f2_fma(v, x[2], g[13]); } \
      { const unsigned long long p = f2_mul(x[2], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(258), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } { const unsigned long long s = f2_mul(W(357), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[2] = f2_fma(v, x[14], g[2]); g[14] = f2_fma(v, x[2], g[14]); } \
      { const unsigned long long p = f2_mul(x[2], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(259), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[2] = f2_fma(v, x[15], g[2]); g[15] = f2_fma(v, x[2], g[15]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); unsigned long long v; v = f2_mul(W(4), adj[0]); { const unsigned long long s = f2_mul(W(358), adj[3]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(52), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(53), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(156), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(157), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(260), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(359), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(261), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(360), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[3], g[3]); g[3] = f2_fma(v, x[3], g[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); unsigned long long v; v = f2_mul(W(99), adj[1]); { const unsigned long long s = f2_mul(W(361), adj[3]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(262), adj[2]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(158), adj[1]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(159), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(54), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(55), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[3] = f2_fma(v, x[4], g[3]); g[4] = f2_fma(v, x[3], g[4]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(362), adj[3]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } { const unsigned long long s = f2_mul(W(160), adj[1]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(56), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } g[3] = f2_fma(v, x[5], g[3]); g[5] = f2_fma(v, x[3], g[5]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); unsigned long long v; v = f2_mul(W(308), adj[3]); { const unsigned long long s = f2_mul(W(363), adj[3]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(263), adj[2]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(364), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(57), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[3] = f2_fma(v, x[6], g[3]); g[6] = f2_fma(v, x[3], g[6]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); unsigned long long v; v = f2_mul(W(216), adj[2]); { const unsigned long long s = f2_mul(W(365), adj[3]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(264), adj[2]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(58), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(59), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[3] = f2_fma(v, x[7], g[3]); g[7] = f2_fma(v, x[3], g[7]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); unsigned long long v; v = f2_mul(W(309), adj[3]); { const unsigned long long s = f2_mul(W(366), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(60), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(61), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[8], g[3]); g[8] = f2_fma(v, x[3], g[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(367), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(265), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(368), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(161), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(162), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[9], g[3]); g[9] = f2_fma(v, x[3], g[9]); } \
      { const unsigned long long p = f2_mul(x[3], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(369), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(266), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(163), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(164), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[3] = f2_fma(v, x[10], g[3]); g[10] = f2_fma(v, x[3], g[10]); } \
      { const unsigned long long p = f2_mul(x[3], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(370), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } { const unsigned long long s = f2_mul(W(165), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(166), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[11], g[3]); g[11] = f2_fma(v, x[3], g[11]); } \
      { const unsigned long long p = f2_mul(x[3], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(371), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(267), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(372), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[3] = f2_fma(v, x[12], g[3]); g[12] = f2_fma(v, x[3], g[12]); } \
      { const unsigned long long p = f2_mul(x[3], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(373), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(268), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(374), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[13], g[3]); g[13] = f2_fma(v, x[3], g[13]); } \
      { const unsigned long long p = f2_mul(x[3], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(375), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } { const unsigned long long s = f2_mul(W(269), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[14], g[3]); g[14] = f2_fma(v, x[3], g[14]); } \
      { const unsigned long long p = f2_mul(x[3], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(376), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[3] = f2_fma(v, x[15], g[3]); g[15] = f2_fma(v, x[3], g[15]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); unsigned long long v; v = f2_mul(W(5), adj[0]); { const unsigned long long s = f2_mul(W(62), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(167), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(168), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(270), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(377), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(378), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[4], g[4]); g[4] = f2_fma(v, x[4], g[4]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(63), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } { const unsigned long long s = f2_mul(W(169), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(379), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(271), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(380), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(272), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[5], g[4]); g[5] = f2_fma(v, x[4], g[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(381), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(273), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(382), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(170), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(171), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[6], g[4]); g[6] = f2_fma(v, x[4], g[6]); } \
      { const unsigned long long p = f2_mul(x[4], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(274), adj[2]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(383), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(275), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(172), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(173), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[4] = f2_fma(v, x[7], g[4]); g[7] = f2_fma(v, x[4], g[7]); } \
      { const unsigned long long p = f2_mul(x[4], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(384), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(385), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(174), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(175), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[8], g[4]); g[8] = f2_fma(v, x[4], g[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); unsigned long long v; v = f2_mul(W(310), adj[3]); { const unsigned long long s = f2_mul(W(64), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[4] = f2_fma(v, x[9], g[4]); g[9] = f2_fma(v, x[4], g[9]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); unsigned long long v; v = f2_mul(W(217), adj[2]); { const unsigned long long s = f2_mul(W(65), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } g[4] = f2_fma(v, x[10], g[4]); g[10] = f2_fma(v, x[4], g[10]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); unsigned long long v; v = f2_mul(W(311), adj[3]); { const unsigned long long s = f2_mul(W(66), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(67), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[11], g[4]); g[11] = f2_fma(v, x[4], g[11]); } \
      { unsigned long long v; v = f2_mul(W(100), adj[1]); g[4] = f2_fma(v, x[13], g[4]); g[13] = f2_fma(v, x[4], g[13]); } \
      { unsigned long long v; v = f2_mul(W(101), adj[1]); g[4] = f2_fma(v, x[15], g[4]); g[15] = f2_fma(v, x[4], g[15]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); unsigned long long v; v = f2_mul(W(6), adj[0]); { const unsigned long long s = f2_mul(W(68), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(69), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(176), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(177), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(276), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(386), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(277), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(387), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[5], g[5]); g[5] = f2_fma(v, x[5], g[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(388), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(278), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(178), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(179), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[6], g[5]); g[6] = f2_fma(v, x[5], g[6]); } \
      { const unsigned long long p = f2_mul(x[5], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(389), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(279), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(390), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(180), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(181), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[7], g[5]); g[7] = f2_fma(v, x[5], g[7]); } \
      { const unsigned long long p = f2_mul(x[5], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(280), adj[2]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(391), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(281), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(182), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(183), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[8], g[5]); g[8] = f2_fma(v, x[5], g[8]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(70), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[5] = f2_fma(v, x[9], g[5]); g[9] = f2_fma(v, x[5], g[9]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); unsigned long long v; v = f2_mul(W(312), adj[3]); { const unsigned long long s = f2_mul(W(71), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(72), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[10], g[5]); g[10] = f2_fma(v, x[5], g[10]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); unsigned long long v; v = f2_mul(W(218), adj[2]); { const unsigned long long s = f2_mul(W(73), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(74), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[11], g[5]); g[11] = f2_fma(v, x[5], g[11]); } \
      { unsigned long long v; v = f2_mul(W(102), adj[1]); g[5] = f2_fma(v, x[12], g[5]); g[12] = f2_fma(v, x[5], g[12]); } \
      { unsigned long long v; v = f2_mul(W(103), adj[1]); g[5] = f2_fma(v, x[14], g[5]); g[14] = f2_fma(v, x[5], g[14]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); unsigned long long v; v = f2_mul(W(7), adj[0]); { const unsigned long long s = f2_mul(W(75), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(184), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(282), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(392), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[6] = f2_fma(v, x[6], g[6]); g[6] = f2_fma(v, x[6], g[6]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(76), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } { const unsigned long long s = f2_mul(W(185), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(393), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(283), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(394), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[6] = f2_fma(v, x[7], g[6]); g[7] = f2_fma(v, x[6], g[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(77), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } { const unsigned long long s = f2_mul(W(186), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(187), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(395), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(284), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(396), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[6] = f2_fma(v, x[8], g[6]); g[8] = f2_fma(v, x[6], g[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(78), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[6] = f2_fma(v, x[9], g[6]); g[9] = f2_fma(v, x[6], g[9]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); unsigned long long v; v = f2_mul(W(104), adj[1]); { const unsigned long long s = f2_mul(W(79), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[6] = f2_fma(v, x[11], g[6]); g[11] = f2_fma(v, x[6], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); unsigned long long v; v = f2_mul(W(219), adj[2]); { const unsigned long long s = f2_mul(W(80), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } g[6] = f2_fma(v, x[12], g[6]); g[12] = f2_fma(v, x[6], g[12]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); unsigned long long v; v = f2_mul(W(313), adj[3]); { const unsigned long long s = f2_mul(W(81), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[6] = f2_fma(v, x[13], g[6]); g[13] = f2_fma(v, x[6], g[13]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(82), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[6] = f2_fma(v, x[15], g[6]); g[15] = f2_fma(v, x[6], g[15]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); unsigned long long v; v = f2_mul(W(8), adj[0]); { const unsigned long long s = f2_mul(W(83), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(188), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(189), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(285), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(397), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(286), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(398), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[7], g[7]); g[7] = f2_fma(v, x[7], g[7]); } \
      { const unsigned long long p = f2_mul(x[7], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(190), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(399), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(287), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(400), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(288), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[8], g[7]); g[8] = f2_fma(v, x[7], g[8]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(84), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[7] = f2_fma(v, x[9], g[7]); g[9] = f2_fma(v, x[7], g[9]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); unsigned long long v; v = f2_mul(W(105), adj[1]); { const unsigned long long s = f2_mul(W(85), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[7] = f2_fma(v, x[10], g[7]); g[10] = f2_fma(v, x[7], g[10]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); unsigned long long v; v = f2_mul(W(314), adj[3]); { const unsigned long long s = f2_mul(W(86), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[7] = f2_fma(v, x[12], g[7]); g[12] = f2_fma(v, x[7], g[12]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); unsigned long long v; v = f2_mul(W(220), adj[2]); { const unsigned long long s = f2_mul(W(87), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[7] = f2_fma(v, x[13], g[7]); g[13] = f2_fma(v, x[7], g[13]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); unsigned long long v; v = f2_mul(W(315), adj[3]); { const unsigned long long s = f2_mul(W(88), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[14], g[7]); g[14] = f2_fma(v, x[7], g[14]); } \
      { const unsigned long long p = f2_mul(x[8], x[8]); unsigned long long v; v = f2_mul(W(9), adj[0]); { const unsigned long long s = f2_mul(W(191), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(192), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(289), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(401), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(402), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[8], g[8]); g[8] = f2_fma(v, x[8], g[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); unsigned long long v; v = f2_mul(W(106), adj[1]); { const unsigned long long s = f2_mul(W(89), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[8] = f2_fma(v, x[9], g[8]); g[9] = f2_fma(v, x[8], g[9]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); unsigned long long v; v = f2_mul(W(107), adj[1]); { const unsigned long long s = f2_mul(W(90), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[8] = f2_fma(v, x[11], g[8]); g[11] = f2_fma(v, x[8], g[11]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(91), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[8] = f2_fma(v, x[12], g[8]); g[12] = f2_fma(v, x[8], g[12]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); unsigned long long v; v = f2_mul(W(316), adj[3]); { const unsigned long long s = f2_mul(W(92), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(93), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[13], g[8]); g[13] = f2_fma(v, x[8], g[13]); } \
      { unsigned long long v; v = f2_mul(W(221), adj[2]); g[8] = f2_fma(v, x[14], g[8]); g[14] = f2_fma(v, x[8], g[14]); } \
      { unsigned long long v; v = f2_mul(W(317), adj[3]); g[8] = f2_fma(v, x[15], g[8]); g[15] = f2_fma(v, x[8], g[15]); } \
      { const unsigned long long p = f2_mul(x[9], x[9]); unsigned long long v; v = f2_mul(W(10), adj[0]); { const unsigned long long s = f2_mul(W(193), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(290), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(403), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[9] = f2_fma(v, x[9], g[9]); g[9] = f2_fma(v, x[9], g[9]); } \
      { const unsigned long long p = f2_mul(x[9], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(194), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(404), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(291), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(405), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[9] = f2_fma(v, x[10], g[9]); g[10] = f2_fma(v, x[9], g[10]); } \
      { const unsigned long long p = f2_mul(x[9], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(195), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } { const unsigned long long s = f2_mul(W(406), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(292), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(407), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[9] = f2_fma(v, x[11], g[9]); g[11] = f2_fma(v, x[9], g[11]); } \
      { const unsigned long long p = f2_mul(x[9], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(196), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[9] = f2_fma(v, x[12], g[9]); g[12] = f2_fma(v, x[9], g[12]); } \
      { const unsigned long long p = f2_mul(x[9], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(197), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(198), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[9] = f2_fma(v, x[13], g[9]); g[13] = f2_fma(v, x[9], g[13]); } \
      { const unsigned long long p = f2_mul(x[9], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(199), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[9] = f2_fma(v, x[14], g[9]); g[14] = f2_fma(v, x[9], g[14]); } \
      { const unsigned long long p = f2_mul(x[10], x[10]); unsigned long long v; v = f2_mul(W(11), adj[0]); { const unsigned long long s = f2_mul(W(200), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(293), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(408), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(409), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[10] = f2_fma(v, x[10], g[10]); g[10] = f2_fma(v, x[10], g[10]); } \
      { const unsigned long long p = f2_mul(x[10], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(410), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(294), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(411), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(295), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[10] = f2_fma(v, x[11], g[10]); g[11] = f2_fma(v, x[10], g[11]); } \
      { const unsigned long long p = f2_mul(x[10], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(201), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(202), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[10] = f2_fma(v, x[12], g[10]); g[12] = f2_fma(v, x[10], g[12]); } \
      { const unsigned long long p = f2_mul(x[10], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(203), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[10] = f2_fma(v, x[13], g[10]); g[13] = f2_fma(v, x[10], g[13]); } \
      { const unsigned long long p = f2_mul(x[10], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(204), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[10] = f2_fma(v, x[14], g[10]); g[14] = f2_fma(v, x[10], g[14]); } \
      { const unsigned long long p = f2_mul(x[11], x[11]); unsigned long long v; v = f2_mul(W(12), adj[0]); { const unsigned long long s = f2_mul(W(205), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(296), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(412), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(297), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(413), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[11] = f2_fma(v, x[11], g[11]); g[11] = f2_fma(v, x[11], g[11]); } \
      { const unsigned long long p = f2_mul(x[11], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(206), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(207), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[11] = f2_fma(v, x[12], g[11]); g[12] = f2_fma(v, x[11], g[12]); } \
      { const unsigned long long p = f2_mul(x[11], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(208), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(209), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[11] = f2_fma(v, x[13], g[11]); g[13] = f2_fma(v, x[11], g[13]); } \
      { const unsigned long long p = f2_mul(x[11], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(210), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[11] = f2_fma(v, x[14], g[11]); g[14] = f2_fma(v, x[11], g[14]); } \
      { const unsigned long long p = f2_mul(x[11], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(211), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[11] = f2_fma(v, x[15], g[11]); g[15] = f2_fma(v, x[11], g[15]); } \
      { const unsigned long long p = f2_mul(x[12], x[12]); unsigned long long v; v = f2_mul(W(13), adj[0]); { const unsigned long long s = f2_mul(W(298), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(414), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[12] = f2_fma(v, x[12], g[12]); g[12] = f2_fma(v, x[12], g[12]); } \
      { const unsigned long long p = f2_mul(x[12], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(299), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(415), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[12] = f2_fma(v, x[13], g[12]); g[13] = f2_fma(v, x[12], g[13]); } \
      { const unsigned long long p = f2_mul(x[12], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(300), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } { const unsigned long long s = f2_mul(W(416), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[12] = f2_fma(v, x[14], g[12]); g[14] = f2_fma(v, x[12], g[14]); } \
      { const unsigned long long p = f2_mul(x[12], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(301), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[12] = f2_fma(v, x[15], g[12]); g[15] = f2_fma(v, x[12], g[15]); } \
      { const unsigned long long p = f2_mul(x[13], x[13]); unsigned long long v; v = f2_mul(W(14), adj[0]); { const unsigned long long s = f2_mul(W(417), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(302), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(418), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[13] = f2_fma(v, x[13], g[13]); g[13] = f2_fma(v, x[13], g[13]); } \
      { const unsigned long long p = f2_mul(x[13], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(419), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } { const unsigned long long s = f2_mul(W(303), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[13] = f2_fma(v, x[14], g[13]); g[14] = f2_fma(v, x[13], g[14]); } \
      { const unsigned long long p = f2_mul(x[13], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(420), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[13] = f2_fma(v, x[15], g[13]); g[15] = f2_fma(v, x[13], g[15]); } \
      { const unsigned long long p = f2_mul(x[14], x[14]); unsigned long long v; v = f2_mul(W(15), adj[0]); { const unsigned long long s = f2_mul(W(421), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[14] = f2_fma(v, x[14], g[14]); g[14] = f2_fma(v, x[14], g[14]); } \
      { unsigned long long v; v = f2_mul(W(16), adj[0]); g[15] = f2_fma(v, x[15], g[15]); g[15] = f2_fma(v, x[15], g[15]); }
#define SXB_S1_M1_FORWARD_BODY \
      o[0] = f2_fma(W(0), x[0], o[0]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); o[0] = f2_fma(p, f2_fma(W(17), x[0], W(1)), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); o[0] = f2_fma(p, f2_mul(W(18), x[1]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); o[0] = f2_fma(p, f2_mul(W(19), x[2]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); o[0] = f2_fma(p, f2_mul(W(20), x[3]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); o[0] = f2_fma(p, f2_mul(W(21), x[4]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); o[0] = f2_fma(p, f2_mul(W(22), x[5]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); o[0] = f2_fma(p, f2_mul(W(23), x[6]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); o[0] = f2_fma(p, f2_mul(W(24), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); o[0] = f2_fma(p, f2_mul(W(25), x[8]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); o[0] = f2_fma(p, f2_mul(W(26), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); o[0] = f2_fma(p, f2_mul(W(27), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); o[0] = f2_fma(p, f2_mul(W(28), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); o[0] = f2_fma(p, f2_mul(W(29), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); o[0] = f2_fma(p, f2_mul(W(30), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); o[0] = f2_fma(p, f2_mul(W(31), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); o[0] = f2_fma(p, f2_mul(W(32), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); o[0] = f2_fma(p, f2_fma(W(34), x[8], f2_fma(W(33), x[6], W(2))), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); o[0] = f2_fma(p, f2_mul(W(35), x[5]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); o[0] = f2_fma(p, f2_mul(W(36), x[4]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); o[0] = f2_fma(p, f2_fma(W(38), x[15], f2_mul(W(37), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); o[0] = f2_fma(p, f2_fma(W(40), x[14], f2_mul(W(39), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); o[0] = f2_fma(p, f2_mul(W(41), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); o[0] = f2_fma(p, f2_mul(W(42), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); o[0] = f2_fma(p, f2_fma(W(44), x[11], f2_mul(W(43), x[9])), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); o[0] = f2_fma(p, f2_fma(W(45), x[6], W(3)), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); o[0] = f2_fma(p, f2_mul(W(46), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); o[0] = f2_fma(p, f2_mul(W(47), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); o[0] = f2_fma(p, f2_mul(W(48), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); o[0] = f2_fma(p, f2_mul(W(49), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); o[0] = f2_fma(p, f2_mul(W(50), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); o[0] = f2_fma(p, f2_mul(W(51), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); o[0] = f2_fma(p, f2_fma(W(53), x[8], f2_fma(W(52), x[6], W(4))), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); o[0] = f2_fma(p, f2_fma(W(55), x[11], f2_mul(W(54), x[9])), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); o[0] = f2_fma(p, f2_mul(W(56), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); o[0] = f2_fma(p, f2_mul(W(57), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); o[0] = f2_fma(p, f2_fma(W(59), x[14], f2_mul(W(58), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); o[0] = f2_fma(p, f2_fma(W(61), x[15], f2_mul(W(60), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); o[0] = f2_fma(p, f2_fma(W(62), x[6], W(5)), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); o[0] = f2_fma(p, f2_mul(W(63), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); o[0] = f2_fma(p, f2_mul(W(64), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); o[0] = f2_fma(p, f2_mul(W(65), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); o[0] = f2_fma(p, f2_fma(W(67), x[15], f2_mul(W(66), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); o[0] = f2_fma(p, f2_fma(W(69), x[8], f2_fma(W(68), x[6], W(6))), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); o[0] = f2_fma(p, f2_mul(W(70), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); o[0] = f2_fma(p, f2_fma(W(72), x[15], f2_mul(W(71), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); o[0] = f2_fma(p, f2_fma(W(74), x[14], f2_mul(W(73), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); o[0] = f2_fma(p, f2_fma(W(75), x[6], W(7)), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); o[0] = f2_fma(p, f2_mul(W(76), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); o[0] = f2_fma(p, f2_mul(W(77), x[8]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); o[0] = f2_fma(p, f2_mul(W(78), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); o[0] = f2_fma(p, f2_mul(W(79), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); o[0] = f2_fma(p, f2_mul(W(80), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); o[0] = f2_fma(p, f2_mul(W(81), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); o[0] = f2_fma(p, f2_mul(W(82), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); o[0] = f2_fma(p, f2_fma(W(83), x[8], W(8)), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); o[0] = f2_fma(p, f2_mul(W(84), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); o[0] = f2_fma(p, f2_mul(W(85), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); o[0] = f2_fma(p, f2_mul(W(86), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); o[0] = f2_fma(p, f2_mul(W(87), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); o[0] = f2_fma(p, f2_mul(W(88), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[8]); o[0] = f2_fma(p, W(9), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); o[0] = f2_fma(p, f2_mul(W(89), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); o[0] = f2_fma(p, f2_mul(W(90), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); o[0] = f2_fma(p, f2_mul(W(91), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); o[0] = f2_fma(p, f2_fma(W(93), x[15], f2_mul(W(92), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[9], x[9]); o[0] = f2_fma(p, W(10), o[0]); } \
      { const unsigned long long p = f2_mul(x[10], x[10]); o[0] = f2_fma(p, W(11), o[0]); } \
      { const unsigned long long p = f2_mul(x[11], x[11]); o[0] = f2_fma(p, W(12), o[0]); } \
      { const unsigned long long p = f2_mul(x[12], x[12]); o[0] = f2_fma(p, W(13), o[0]); } \
      { const unsigned long long p = f2_mul(x[13], x[13]); o[0] = f2_fma(p, W(14), o[0]); } \
      { const unsigned long long p = f2_mul(x[14], x[14]); o[0] = f2_fma(p, W(15), o[0]); } \
      { const unsigned long long p = f2_mul(x[15], x[15]); o[0] = f2_fma(p, W(16), o[0]); }
#define SXB_S1_M1_REVERSE_BODY \
      g[0] = f2_fma(W(0), adj[0], g[0]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); unsigned long long v; v = f2_mul(W(1), adj[0]); { const unsigned long long s = f2_mul(W(17), adj[0]); g[0] = f2_fma(s, p, g[0]); v = f2_fma(s, x[0], v); } g[0] = f2_fma(v, x[0], g[0]); g[0] = f2_fma(v, x[0], g[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); unsigned long long v; { const unsigned long long s = f2_mul(W(18), adj[0]); g[1] = f2_fma(s, p, g[1]); v = f2_mul(s, x[1]); } g[0] = f2_fma(v, x[1], g[0]); g[1] = f2_fma(v, x[0], g[1]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(19), adj[0]); g[2] = f2_fma(s, p, g[2]); v = f2_mul(s, x[2]); } g[0] = f2_fma(v, x[2], g[0]); g[2] = f2_fma(v, x[0], g[2]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(20), adj[0]); g[3] = f2_fma(s, p, g[3]); v = f2_mul(s, x[3]); } g[0] = f2_fma(v, x[3], g[0]); g[3] = f2_fma(v, x[0], g[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(21), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } g[0] = f2_fma(v, x[4], g[0]); g[4] = f2_fma(v, x[0], g[4]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(22), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } g[0] = f2_fma(v, x[5], g[0]); g[5] = f2_fma(v, x[0], g[5]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(23), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_mul(s, x[6]); } g[0] = f2_fma(v, x[6], g[0]); g[6] = f2_fma(v, x[0], g[6]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(24), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[0] = f2_fma(v, x[7], g[0]); g[7] = f2_fma(v, x[0], g[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(25), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } g[0] = f2_fma(v, x[8], g[0]); g[8] = f2_fma(v, x[0], g[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(26), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[0] = f2_fma(v, x[9], g[0]); g[9] = f2_fma(v, x[0], g[9]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(27), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[0] = f2_fma(v, x[10], g[0]); g[10] = f2_fma(v, x[0], g[10]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(28), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[0] = f2_fma(v, x[11], g[0]); g[11] = f2_fma(v, x[0], g[11]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(29), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[0] = f2_fma(v, x[12], g[0]); g[12] = f2_fma(v, x[0], g[12]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(30), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[0] = f2_fma(v, x[13], g[0]); g[13] = f2_fma(v, x[0], g[13]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(31), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[0] = f2_fma(v, x[14], g[0]); g[14] = f2_fma(v, x[0], g[14]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(32), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[0] = f2_fma(v, x[15], g[0]); g[15] = f2_fma(v, x[0], g[15]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); unsigned long long v; v = f2_mul(W(2), adj[0]); { const unsigned long long s = f2_mul(W(33), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(34), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[1] = f2_fma(v, x[1], g[1]); g[1] = f2_fma(v, x[1], g[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(35), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } g[1] = f2_fma(v, x[2], g[1]); g[2] = f2_fma(v, x[1], g[2]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(36), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } g[1] = f2_fma(v, x[3], g[1]); g[3] = f2_fma(v, x[1], g[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(37), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(38), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[4], g[1]); g[4] = f2_fma(v, x[1], g[4]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(39), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(40), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[5], g[1]); g[5] = f2_fma(v, x[1], g[5]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(41), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[1] = f2_fma(v, x[6], g[1]); g[6] = f2_fma(v, x[1], g[6]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(42), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[1] = f2_fma(v, x[7], g[1]); g[7] = f2_fma(v, x[1], g[7]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(43), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(44), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[1] = f2_fma(v, x[8], g[1]); g[8] = f2_fma(v, x[1], g[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); unsigned long long v; v = f2_mul(W(3), adj[0]); { const unsigned long long s = f2_mul(W(45), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[2] = f2_fma(v, x[2], g[2]); g[2] = f2_fma(v, x[2], g[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(46), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[2] = f2_fma(v, x[3], g[2]); g[3] = f2_fma(v, x[2], g[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(47), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[2] = f2_fma(v, x[4], g[2]); g[4] = f2_fma(v, x[2], g[4]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(48), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[2] = f2_fma(v, x[5], g[2]); g[5] = f2_fma(v, x[2], g[5]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(49), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[2] = f2_fma(v, x[6], g[2]); g[6] = f2_fma(v, x[2], g[6]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(50), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[2] = f2_fma(v, x[7], g[2]); g[7] = f2_fma(v, x[2], g[7]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(51), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[2] = f2_fma(v, x[8], g[2]); g[8] = f2_fma(v, x[2], g[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); unsigned long long v; v = f2_mul(W(4), adj[0]); { const unsigned long long s = f2_mul(W(52), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(53), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[3] = f2_fma(v, x[3], g[3]); g[3] = f2_fma(v, x[3], g[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(54), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(55), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[3] = f2_fma(v, x[4], g[3]); g[4] = f2_fma(v, x[3], g[4]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(56), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[3] = f2_fma(v, x[5], g[3]); g[5] = f2_fma(v, x[3], g[5]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(57), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[3] = f2_fma(v, x[6], g[3]); g[6] = f2_fma(v, x[3], g[6]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(58), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(59), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[3] = f2_fma(v, x[7], g[3]); g[7] = f2_fma(v, x[3], g[7]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(60), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(61), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[8], g[3]); g[8] = f2_fma(v, x[3], g[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); unsigned long long v; v = f2_mul(W(5), adj[0]); { const unsigned long long s = f2_mul(W(62), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[4] = f2_fma(v, x[4], g[4]); g[4] = f2_fma(v, x[4], g[4]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(63), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[4] = f2_fma(v, x[5], g[4]); g[5] = f2_fma(v, x[4], g[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(64), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[4] = f2_fma(v, x[9], g[4]); g[9] = f2_fma(v, x[4], g[9]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(65), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[4] = f2_fma(v, x[10], g[4]); g[10] = f2_fma(v, x[4], g[10]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(66), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(67), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[11], g[4]); g[11] = f2_fma(v, x[4], g[11]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); unsigned long long v; v = f2_mul(W(6), adj[0]); { const unsigned long long s = f2_mul(W(68), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(69), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[5] = f2_fma(v, x[5], g[5]); g[5] = f2_fma(v, x[5], g[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(70), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[5] = f2_fma(v, x[9], g[5]); g[9] = f2_fma(v, x[5], g[9]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(71), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(72), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[10], g[5]); g[10] = f2_fma(v, x[5], g[10]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(73), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(74), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[11], g[5]); g[11] = f2_fma(v, x[5], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); unsigned long long v; v = f2_mul(W(7), adj[0]); { const unsigned long long s = f2_mul(W(75), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[6] = f2_fma(v, x[6], g[6]); g[6] = f2_fma(v, x[6], g[6]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(76), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[6] = f2_fma(v, x[7], g[6]); g[7] = f2_fma(v, x[6], g[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(77), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } g[6] = f2_fma(v, x[8], g[6]); g[8] = f2_fma(v, x[6], g[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(78), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[6] = f2_fma(v, x[9], g[6]); g[9] = f2_fma(v, x[6], g[9]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(79), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[6] = f2_fma(v, x[11], g[6]); g[11] = f2_fma(v, x[6], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(80), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[6] = f2_fma(v, x[12], g[6]); g[12] = f2_fma(v, x[6], g[12]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(81), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[6] = f2_fma(v, x[13], g[6]); g[13] = f2_fma(v, x[6], g[13]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(82), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[6] = f2_fma(v, x[15], g[6]); g[15] = f2_fma(v, x[6], g[15]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); unsigned long long v; v = f2_mul(W(8), adj[0]); { const unsigned long long s = f2_mul(W(83), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[7] = f2_fma(v, x[7], g[7]); g[7] = f2_fma(v, x[7], g[7]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(84), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[7] = f2_fma(v, x[9], g[7]); g[9] = f2_fma(v, x[7], g[9]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(85), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[7] = f2_fma(v, x[10], g[7]); g[10] = f2_fma(v, x[7], g[10]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(86), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[7] = f2_fma(v, x[12], g[7]); g[12] = f2_fma(v, x[7], g[12]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(87), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[7] = f2_fma(v, x[13], g[7]); g[13] = f2_fma(v, x[7], g[13]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(88), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[7] = f2_fma(v, x[14], g[7]); g[14] = f2_fma(v, x[7], g[14]); } \
      { unsigned long long v; v = f2_mul(W(9), adj[0]); g[8] = f2_fma(v, x[8], g[8]); g[8] = f2_fma(v, x[8], g[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(89), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[8] = f2_fma(v, x[9], g[8]); g[9] = f2_fma(v, x[8], g[9]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(90), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[8] = f2_fma(v, x[11], g[8]); g[11] = f2_fma(v, x[8], g[11]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(91), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[8] = f2_fma(v, x[12], g[8]); g[12] = f2_fma(v, x[8], g[12]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(92), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(93), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[13], g[8]); g[13] = f2_fma(v, x[8], g[13]); } \
      { unsigned long long v; v = f2_mul(W(10), adj[0]); g[9] = f2_fma(v, x[9], g[9]); g[9] = f2_fma(v, x[9], g[9]); } \
      { unsigned long long v; v = f2_mul(W(11), adj[0]); g[10] = f2_fma(v, x[10], g[10]); g[10] = f2_fma(v, x[10], g[10]); } \
      { unsigned long long v; v = f2_mul(W(12), adj[0]); g[11] = f2_fma(v, x[11], g[11]); g[11] = f2_fma(v, x[11], g[11]); } \
      { unsigned long long v; v = f2_mul(W(13), adj[0]); g[12] = f2_fma(v, x[12], g[12]); g[12] = f2_fma(v, x[12], g[12]); } \
      { unsigned long long v; v = f2_mul(W(14), adj[0]); g[13] = f2_fma(v, x[13], g[13]); g[13] = f2_fma(v, x[13], g[13]); } \
      { unsigned long long v; v = f2_mul(W(15), adj[0]); g[14] = f2_fma(v, x[14], g[14]); g[14] = f2_fma(v, x[14], g[14]); } \
      { unsigned long long v; v = f2_mul(W(16), adj[0]); g[15] = f2_fma(v, x[15], g[15]); g[15] = f2_fma(v, x[15], g[15]); }
#define SXB_S1_L1_FORWARD_BODY \
    { /* path 0: edge l=0, source l=0 -> l=0 */ \
      const float t0 = R[0] * h[0]; \
      acc[0] = fmaf(t0, y[0], acc[0]); \
    } \
    { /* path 1: edge l=1, source l=1 -> l=0 */ \
      const float t0 = R[1] * h[1]; \
      const float t1 = R[1] * h[2]; \
      const float t2 = R[1] * h[3]; \
      acc[1] = fmaf(t0, y[1], acc[1]); \
      acc[2] = fmaf(t1, y[1], acc[2]); \
      acc[3] = fmaf(t2, y[1], acc[3]); \
      acc[4] = fmaf(t0, y[2], acc[4]); \
      acc[5] = fmaf(t1, y[2], acc[5]); \
      acc[6] = fmaf(t2, y[2], acc[6]); \
      acc[7] = fmaf(t0, y[3], acc[7]); \
      acc[8] = fmaf(t1, y[3], acc[8]); \
      acc[9] = fmaf(t2, y[3], acc[9]); \
    } \
    { /* path 2: edge l=1, source l=0 -> l=1 */ \
      const float t0 = R[2] * h[0]; \
      acc[10] = fmaf(t0, y[1], acc[10]); \
      acc[11] = fmaf(t0, y[2], acc[11]); \
      acc[12] = fmaf(t0, y[3], acc[12]); \
    } \
    { /* path 3: edge l=0, source l=1 -> l=1 */ \
      const float t0 = R[3] * h[1]; \
      const float t1 = R[3] * h[2]; \
      const float t2 = R[3] * h[3]; \
      acc[13] = fmaf(t0, y[0], acc[13]); \
      acc[14] = fmaf(t1, y[0], acc[14]); \
      acc[15] = fmaf(t2, y[0], acc[15]); \
    } \
    { /* path 4: edge l=2, source l=1 -> l=1 */ \
      const float t0 = R[4] * h[1]; \
      const float t1 = R[4] * h[2]; \
      const float t2 = R[4] * h[3]; \
      acc[16] = fmaf(t0, y[4], acc[16]); \
      acc[17] = fmaf(t1, y[4], acc[17]); \
      acc[18] = fmaf(t2, y[4], acc[18]); \
      acc[19] = fmaf(t0, y[5], acc[19]); \
      acc[20] = fmaf(t1, y[5], acc[20]); \
      acc[21] = fmaf(t2, y[5], acc[21]); \
      acc[22] = fmaf(t0, y[6], acc[22]); \
      acc[23] = fmaf(t1, y[6], acc[23]); \
      acc[24] = fmaf(t2, y[6], acc[24]); \
      acc[25] = fmaf(t0, y[7], acc[25]); \
      acc[26] = fmaf(t1, y[7], acc[26]); \
      acc[27] = fmaf(t2, y[7], acc[27]); \
      acc[28] = fmaf(t0, y[8], acc[28]); \
      acc[29] = fmaf(t1, y[8], acc[29]); \
      acc[30] = fmaf(t2, y[8], acc[30]); \
    } \
    { /* path 5: edge l=2, source l=0 -> l=2 */ \
      const float t0 = R[5] * h[0]; \
      acc[31] = fmaf(t0, y[4], acc[31]); \
      acc[32] = fmaf(t0, y[5], acc[32]); \
      acc[33] = fmaf(t0, y[6], acc[33]); \
      acc[34] = fmaf(t0, y[7], acc[34]); \
      acc[35] = fmaf(t0, y[8], acc[35]); \
    } \
    { /* path 6: edge l=1, source l=1 -> l=2 */ \
      const float t0 = R[6] * h[1]; \
      const float t1 = R[6] * h[2]; \
      const float t2 = R[6] * h[3]; \
      acc[36] = fmaf(t0, y[1], acc[36]); \
      acc[37] = fmaf(t1, y[1], acc[37]); \
      acc[38] = fmaf(t2, y[1], acc[38]); \
      acc[39] = fmaf(t0, y[2], acc[39]); \
      acc[40] = fmaf(t1, y[2], acc[40]); \
      acc[41] = fmaf(t2, y[2], acc[41]); \
      acc[42] = fmaf(t0, y[3], acc[42]); \
      acc[43] = fmaf(t1, y[3], acc[43]); \
      acc[44] = fmaf(t2, y[3], acc[44]); \
    } \
    { /* path 7: edge l=3, source l=1 -> l=2 */ \
      const float t0 = R[7] * h[1]; \
      const float t1 = R[7] * h[2]; \
      const float t2 = R[7] * h[3]; \
      acc[45] = fmaf(t0, y[9], acc[45]); \
      acc[46] = fmaf(t1, y[9], acc[46]); \
      acc[47] = fmaf(t2, y[9], acc[47]); \
      acc[48] = fmaf(t0, y[10], acc[48]); \
      acc[49] = fmaf(t1, y[10], acc[49]); \
      acc[50] = fmaf(t2, y[10], acc[50]); \
      acc[51] = fmaf(t0, y[11], acc[51]); \
      acc[52] = fmaf(t1, y[11], acc[52]); \
      acc[53] = fmaf(t2, y[11], acc[53]); \
      acc[54] = fmaf(t0, y[12], acc[54]); \
      acc[55] = fmaf(t1, y[12], acc[55]); \
      acc[56] = fmaf(t2, y[12], acc[56]); \
      acc[57] = fmaf(t0, y[13], acc[57]); \
      acc[58] = fmaf(t1, y[13], acc[58]); \
      acc[59] = fmaf(t2, y[13], acc[59]); \
      acc[60] = fmaf(t0, y[14], acc[60]); \
      acc[61] = fmaf(t1, y[14], acc[61]); \
      acc[62] = fmaf(t2, y[14], acc[62]); \
      acc[63] = fmaf(t0, y[15], acc[63]); \
      acc[64] = fmaf(t1, y[15], acc[64]); \
      acc[65] = fmaf(t2, y[15], acc[65]); \
    } \
    { /* path 8: edge l=3, source l=0 -> l=3 */ \
      const float t0 = R[8] * h[0]; \
      acc[66] = fmaf(t0, y[9], acc[66]); \
      acc[67] = fmaf(t0, y[10], acc[67]); \
      acc[68] = fmaf(t0, y[11], acc[68]); \
      acc[69] = fmaf(t0, y[12], acc[69]); \
      acc[70] = fmaf(t0, y[13], acc[70]); \
      acc[71] = fmaf(t0, y[14], acc[71]); \
      acc[72] = fmaf(t0, y[15], acc[72]); \
    } \
    { /* path 9: edge l=2, source l=1 -> l=3 */ \
      const float t0 = R[9] * h[1]; \
      const float t1 = R[9] * h[2]; \
      const float t2 = R[9] * h[3]; \
      acc[73] = fmaf(t0, y[4], acc[73]); \
      acc[74] = fmaf(t1, y[4], acc[74]); \
      acc[75] = fmaf(t2, y[4], acc[75]); \
      acc[76] = fmaf(t0, y[5], acc[76]); \
      acc[77] = fmaf(t1, y[5], acc[77]); \
      acc[78] = fmaf(t2, y[5], acc[78]); \
      acc[79] = fmaf(t0, y[6], acc[79]); \
      acc[80] = fmaf(t1, y[6], acc[80]); \
      acc[81] = fmaf(t2, y[6], acc[81]); \
      acc[82] = fmaf(t0, y[7], acc[82]); \
      acc[83] = fmaf(t1, y[7], acc[83]); \
      acc[84] = fmaf(t2, y[7], acc[84]); \
      acc[85] = fmaf(t0, y[8], acc[85]); \
      acc[86] = fmaf(t1, y[8], acc[86]); \
      acc[87] = fmaf(t2, y[8], acc[87]); \
    }
#define SXB_S1_L1_REVERSE_BODY \
    { /* path 0: edge l=0, source l=0 -> l=0 */ \
      float yw = 0.0f; \
      const float ry0 = R[0] * y[0]; \
      { const float w = h[0] * adj[0]; \
        ang[0] = fmaf(R[0], w, ang[0]); yw = fmaf(y[0], w, yw); } \
      hadj[0] = fmaf(ry0, adj[0], hadj[0]); \
      radial = fmaf(dR[0], yw, radial); \
    } \
    { /* path 1: edge l=1, source l=1 -> l=0 */ \
      float yw = 0.0f; \
      const float ry0 = R[1] * y[1]; \
      const float ry1 = R[1] * y[2]; \
      const float ry2 = R[1] * y[3]; \
      { const float w = h[1] * adj[1]; \
        ang[1] = fmaf(R[1], w, ang[1]); yw = fmaf(y[1], w, yw); } \
      { const float w = h[2] * adj[5]; \
        ang[2] = fmaf(R[1], w, ang[2]); yw = fmaf(y[2], w, yw); } \
      { const float w = h[3] * adj[9]; \
        ang[3] = fmaf(R[1], w, ang[3]); yw = fmaf(y[3], w, yw); } \
      hadj[1] = fmaf(ry0, adj[1], hadj[1]); \
      hadj[2] = fmaf(ry1, adj[5], hadj[2]); \
      hadj[3] = fmaf(ry2, adj[9], hadj[3]); \
      radial = fmaf(dR[1], yw, radial); \
    } \
    { /* path 2: edge l=1, source l=0 -> l=1 */ \
      float yw = 0.0f; \
      const float rh0 = R[2] * h[0]; \
      ang[1] = fmaf(rh0, adj[10], ang[1]); \
      ang[2] = fmaf(rh0, adj[11], ang[2]); \
      ang[3] = fmaf(rh0, adj[12], ang[3]); \
      { const float s_ = fmaf(y[3], adj[12], fmaf(y[2], adj[11], y[1] * adj[10])); \
        hadj[0] = fmaf(R[2], s_, hadj[0]); yw = fmaf(h[0], s_, yw); } \
      radial = fmaf(dR[2], yw, radial); \
    } \
    { /* path 3: edge l=0, source l=1 -> l=1 */ \
      float yw = 0.0f; \
      const float ry0 = R[3] * y[0]; \
      { const float w = fmaf(h[3], adj[15], fmaf(h[2], adj[14], h[1] * adj[13])); \
        ang[0] = fmaf(R[3], w, ang[0]); yw = fmaf(y[0], w, yw); } \
      hadj[1] = fmaf(ry0, adj[13], hadj[1]); \
      hadj[2] = fmaf(ry0, adj[14], hadj[2]); \
      hadj[3] = fmaf(ry0, adj[15], hadj[3]); \
      radial = fmaf(dR[3], yw, radial); \
    } \
    { /* path 4: edge l=2, source l=1 -> l=1 */ \
      float yw = 0.0f; \
      const float rh0 = R[4] * h[1]; \
      const float rh1 = R[4] * h[2]; \
      const float rh2 = R[4] * h[3]; \
      ang[4] = fmaf(rh0, adj[16], ang[4]); \
      ang[4] = fmaf(rh2, adj[18], ang[4]); \
      ang[5] = fmaf(rh0, adj[19], ang[5]); \
      ang[5] = fmaf(rh1, adj[20], ang[5]); \
      ang[6] = fmaf(rh0, adj[22], ang[6]); \
      ang[6] = fmaf(rh1, adj[23], ang[6]); \
      ang[6] = fmaf(rh2, adj[24], ang[6]); \
      ang[7] = fmaf(rh1, adj[26], ang[7]); \
      ang[7] = fmaf(rh2, adj[27], ang[7]); \
      ang[8] = fmaf(rh0, adj[28], ang[8]); \
      ang[8] = fmaf(rh2, adj[30], ang[8]); \
      { const float s_ = fmaf(y[8], adj[28], fmaf(y[6], adj[22], fmaf(y[5], adj[19], y[4] * adj[16]))); \
        hadj[1] = fmaf(R[4], s_, hadj[1]); yw = fmaf(h[1], s_, yw); } \
      { const float s_ = fmaf(y[7], adj[26], fmaf(y[6], adj[23], y[5] * adj[20])); \
        hadj[2] = fmaf(R[4], s_, hadj[2]); yw = fmaf(h[2], s_, yw); } \
      { const float s_ = fmaf(y[8], adj[30], fmaf(y[7], adj[27], fmaf(y[6], adj[24], y[4] * adj[18]))); \
        hadj[3] = fmaf(R[4], s_, hadj[3]); yw = fmaf(h[3], s_, yw); } \
      radial = fmaf(dR[4], yw, radial); \
    } \
    { /* path 5: edge l=2, source l=0 -> l=2 */ \
      float yw = 0.0f; \
      const float rh0 = R[5] * h[0]; \
      ang[4] = fmaf(rh0, adj[31], ang[4]); \
      ang[5] = fmaf(rh0, adj[32], ang[5]); \
      ang[6] = fmaf(rh0, adj[33], ang[6]); \
      ang[7] = fmaf(rh0, adj[34], ang[7]); \
      ang[8] = fmaf(rh0, adj[35], ang[8]); \
      { const float s_ = fmaf(y[8], adj[35], fmaf(y[7], adj[34], fmaf(y[6], adj[33], fmaf(y[5], adj[32], y[4] * adj[31])))); \
        hadj[0] = fmaf(R[5], s_, hadj[0]); yw = fmaf(h[0], s_, yw); } \
      radial = fmaf(dR[5], yw, radial); \
    } \
    { /* path 6: edge l=1, source l=1 -> l=2 */ \
      float yw = 0.0f; \
      const float ry0 = R[6] * y[1]; \
      const float ry1 = R[6] * y[2]; \
      const float ry2 = R[6] * y[3]; \
      { const float w = fmaf(h[3], adj[38], fmaf(h[2], adj[37], h[1] * adj[36])); \
        ang[1] = fmaf(R[6], w, ang[1]); yw = fmaf(y[1], w, yw); } \
      { const float w = fmaf(h[3], adj[41], fmaf(h[2], adj[40], h[1] * adj[39])); \
        ang[2] = fmaf(R[6], w, ang[2]); yw = fmaf(y[2], w, yw); } \
      { const float w = fmaf(h[3], adj[44], fmaf(h[2], adj[43], h[1] * adj[42])); \
        ang[3] = fmaf(R[6], w, ang[3]); yw = fmaf(y[3], w, yw); } \
      hadj[1] = fmaf(ry0, adj[36], hadj[1]); \
      hadj[1] = fmaf(ry1, adj[39], hadj[1]); \
      hadj[1] = fmaf(ry2, adj[42], hadj[1]); \
      hadj[2] = fmaf(ry0, adj[37], hadj[2]); \
      hadj[2] = fmaf(ry1, adj[40], hadj[2]); \
      hadj[2] = fmaf(ry2, adj[43], hadj[2]); \
      hadj[3] = fmaf(ry0, adj[38], hadj[3]); \
      hadj[3] = fmaf(ry1, adj[41], hadj[3]); \
      hadj[3] = fmaf(ry2, adj[44], hadj[3]); \
      radial = fmaf(dR[6], yw, radial); \
    } \
    { /* path 7: edge l=3, source l=1 -> l=2 */ \
      float yw = 0.0f; \
      const float rh0 = R[7] * h[1]; \
      const float rh1 = R[7] * h[2]; \
      const float rh2 = R[7] * h[3]; \
      ang[9] = fmaf(rh0, adj[45], ang[9]); \
      ang[9] = fmaf(rh2, adj[47], ang[9]); \
      ang[10] = fmaf(rh0, adj[48], ang[10]); \
      ang[10] = fmaf(rh1, adj[49], ang[10]); \
      ang[10] = fmaf(rh2, adj[50], ang[10]); \
      ang[11] = fmaf(rh0, adj[51], ang[11]); \
      ang[11] = fmaf(rh1, adj[52], ang[11]); \
      ang[11] = fmaf(rh2, adj[53], ang[11]); \
      ang[12] = fmaf(rh0, adj[54], ang[12]); \
      ang[12] = fmaf(rh1, adj[55], ang[12]); \
      ang[12] = fmaf(rh2, adj[56], ang[12]); \
      ang[13] = fmaf(rh0, adj[57], ang[13]); \
      ang[13] = fmaf(rh1, adj[58], ang[13]); \
      ang[13] = fmaf(rh2, adj[59], ang[13]); \
      ang[14] = fmaf(rh0, adj[60], ang[14]); \
      ang[14] = fmaf(rh1, adj[61], ang[14]); \
      ang[14] = fmaf(rh2, adj[62], ang[14]); \
      ang[15] = fmaf(rh0, adj[63], ang[15]); \
      ang[15] = fmaf(rh2, adj[65], ang[15]); \
      { const float s_ = fmaf(y[15], adj[63], fmaf(y[14], adj[60], fmaf(y[13], adj[57], fmaf(y[12], adj[54], fmaf(y[11], adj[51], fmaf(y[10], adj[48], y[9] * adj[45])))))); \
        hadj[1] = fmaf(R[7], s_, hadj[1]); yw = fmaf(h[1], s_, yw); } \
      { const float s_ = fmaf(y[14], adj[61], fmaf(y[13], adj[58], fmaf(y[12], adj[55], fmaf(y[11], adj[52], y[10] * adj[49])))); \
        hadj[2] = fmaf(R[7], s_, hadj[2]); yw = fmaf(h[2], s_, yw); } \
      { const float s_ = fmaf(y[15], adj[65], fmaf(y[14], adj[62], fmaf(y[13], adj[59], fmaf(y[12], adj[56], fmaf(y[11], adj[53], fmaf(y[10], adj[50], y[9] * adj[47])))))); \
        hadj[3] = fmaf(R[7], s_, hadj[3]); yw = fmaf(h[3], s_, yw); } \
      radial = fmaf(dR[7], yw, radial); \
    } \
    { /* path 8: edge l=3, source l=0 -> l=3 */ \
      float yw = 0.0f; \
      const float rh0 = R[8] * h[0]; \
      ang[9] = fmaf(rh0, adj[66], ang[9]); \
      ang[10] = fmaf(rh0, adj[67], ang[10]); \
      ang[11] = fmaf(rh0, adj[68], ang[11]); \
      ang[12] = fmaf(rh0, adj[69], ang[12]); \
      ang[13] = fmaf(rh0, adj[70], ang[13]); \
      ang[14] = fmaf(rh0, adj[71], ang[14]); \
      ang[15] = fmaf(rh0, adj[72], ang[15]); \
      { const float s_ = fmaf(y[15], adj[72], fmaf(y[14], adj[71], fmaf(y[13], adj[70], fmaf(y[12], adj[69], fmaf(y[11], adj[68], fmaf(y[10], adj[67], y[9] * adj[66])))))); \
        hadj[0] = fmaf(R[8], s_, hadj[0]); yw = fmaf(h[0], s_, yw); } \
      radial = fmaf(dR[8], yw, radial); \
    } \
    { /* path 9: edge l=2, source l=1 -> l=3 */ \
      float yw = 0.0f; \
      const float rh0 = R[9] * h[1]; \
      const float rh1 = R[9] * h[2]; \
      const float rh2 = R[9] * h[3]; \
      ang[4] = fmaf(rh0, adj[73], ang[4]); \
      ang[4] = fmaf(rh1, adj[74], ang[4]); \
      ang[4] = fmaf(rh2, adj[75], ang[4]); \
      ang[5] = fmaf(rh0, adj[76], ang[5]); \
      ang[5] = fmaf(rh1, adj[77], ang[5]); \
      ang[5] = fmaf(rh2, adj[78], ang[5]); \
      ang[6] = fmaf(rh0, adj[79], ang[6]); \
      ang[6] = fmaf(rh1, adj[80], ang[6]); \
      ang[6] = fmaf(rh2, adj[81], ang[6]); \
      ang[7] = fmaf(rh0, adj[82], ang[7]); \
      ang[7] = fmaf(rh1, adj[83], ang[7]); \
      ang[7] = fmaf(rh2, adj[84], ang[7]); \
      ang[8] = fmaf(rh0, adj[85], ang[8]); \
      ang[8] = fmaf(rh1, adj[86], ang[8]); \
      ang[8] = fmaf(rh2, adj[87], ang[8]); \
      { const float s_ = fmaf(y[8], adj[85], fmaf(y[7], adj[82], fmaf(y[6], adj[79], fmaf(y[5], adj[76], y[4] * adj[73])))); \
        hadj[1] = fmaf(R[9], s_, hadj[1]); yw = fmaf(h[1], s_, yw); } \
      { const float s_ = fmaf(y[8], adj[86], fmaf(y[7], adj[83], fmaf(y[6], adj[80], fmaf(y[5], adj[77], y[4] * adj[74])))); \
        hadj[2] = fmaf(R[9], s_, hadj[2]); yw = fmaf(h[2], s_, yw); } \
      { const float s_ = fmaf(y[8], adj[87], fmaf(y[7], adj[84], fmaf(y[6], adj[81], fmaf(y[5], adj[78], y[4] * adj[75])))); \
        hadj[3] = fmaf(R[9], s_, hadj[3]); yw = fmaf(h[3], s_, yw); } \
      radial = fmaf(dR[9], yw, radial); \
    }
#define SXB_S1_ROW_BATCHES 10
#define SXB_S1_L1_REVERSE_EDGE_BODY \
    { f2 y[1]; load_pair_harmonics<0>(yrow, y); \
    { /* path 0: edge l=0, source l=0 -> l=0 */ RADIAL(0) f2 yw, t[1], v[1]; \
      t[0] = f2_mul(R, y[0]); \
      ROWS(0) { const f2 w = rows[0]; v[0] = f2_mul(h[0], w); hadj[0] = f2_mul(t[0], w); } \
      yw = f2_mul(y[0], v[0]); \
      radial = f2_mul(dR, yw); \
    } \
    { /* path 3: edge l=0, source l=1 -> l=1 */ RADIAL(3) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[1]; v[0] = f2_mul(h[1], w); hadj[1] = f2_mul(t[0], w); } \
      { const f2 w = rows[2]; v[0] = f2_fma(h[2], w, v[0]); hadj[2] = f2_mul(t[0], w); } \
      { const f2 w = rows[3]; v[0] = f2_fma(h[3], w, v[0]); hadj[3] = f2_mul(t[0], w); } \
      yw = f2_mul(y[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
    } \
    { f2 y[3], ang[3]; load_pair_harmonics<1>(yrow, y); \
    { /* path 1: edge l=1, source l=1 -> l=0 */ RADIAL(1) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[4]; v[0] = f2_mul(h[1], w); hadj[1] = f2_fma(t[0], w, hadj[1]); } \
      ang[0] = f2_mul(R, v[0]); yw = f2_mul(y[0], v[0]); \
      t[0] = f2_mul(R, y[1]); \
      { const f2 w = rows[5]; v[0] = f2_mul(h[2], w); hadj[2] = f2_fma(t[0], w, hadj[2]); } \
      ang[1] = f2_mul(R, v[0]); yw = f2_fma(y[1], v[0], yw); \
      t[0] = f2_mul(R, y[2]); \
      { const f2 w = rows[6]; v[0] = f2_mul(h[3], w); hadj[3] = f2_fma(t[0], w, hadj[3]); } \
      ang[2] = f2_mul(R, v[0]); yw = f2_fma(y[2], v[0], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 2: edge l=1, source l=0 -> l=1 */ RADIAL(2) f2 yw, t[1], v[1]; \
      t[0] = f2_mul(R, h[0]); \
      { const f2 w = rows[7]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      ROWS(1) { const f2 w = rows[0]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[1]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      hadj[0] = f2_fma(R, v[0], hadj[0]); yw = f2_mul(h[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 6: edge l=1, source l=1 -> l=2 */ RADIAL(6) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[2]; v[0] = f2_mul(h[1], w); hadj[1] = f2_fma(t[0], w, hadj[1]); } \
      { const f2 w = rows[3]; v[0] = f2_fma(h[2], w, v[0]); hadj[2] = f2_fma(t[0], w, hadj[2]); } \
      { const f2 w = rows[4]; v[0] = f2_fma(h[3], w, v[0]); hadj[3] = f2_fma(t[0], w, hadj[3]); } \
      ang[0] = f2_fma(R, v[0], ang[0]); yw = f2_mul(y[0], v[0]); \
      t[0] = f2_mul(R, y[1]); \
      { const f2 w = rows[5]; v[0] = f2_mul(h[1], w); hadj[1] = f2_fma(t[0], w, hadj[1]); } \
      { const f2 w = rows[6]; v[0] = f2_fma(h[2], w, v[0]); hadj[2] = f2_fma(t[0], w, hadj[2]); } \
      { const f2 w = rows[7]; v[0] = f2_fma(h[3], w, v[0]); hadj[3] = f2_fma(t[0], w, hadj[3]); } \
      ang[1] = f2_fma(R, v[0], ang[1]); yw = f2_fma(y[1], v[0], yw); \
      t[0] = f2_mul(R, y[2]); \
      ROWS(2) { const f2 w = rows[0]; v[0] = f2_mul(h[1], w); hadj[1] = f2_fma(t[0], w, hadj[1]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[2], w, v[0]); hadj[2] = f2_fma(t[0], w, hadj[2]); } \
      { const f2 w = rows[2]; v[0] = f2_fma(h[3], w, v[0]); hadj[3] = f2_fma(t[0], w, hadj[3]); } \
      ang[2] = f2_fma(R, v[0], ang[2]); yw = f2_fma(y[2], v[0], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
      f[1] = f2_sum(ang[0]); f[2] = f2_sum(ang[1]); f[3] = f2_sum(ang[2]); \
    } \
    { f2 y[5], ang[5]; load_pair_harmonics<2>(yrow, y); \
    { /* path 4: edge l=2, source l=1 -> l=1 */ RADIAL(4) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, h[1]); \
      t[1] = f2_mul(R, h[2]); \
      t[2] = f2_mul(R, h[3]); \
      { const f2 w = rows[3]; ang[0] = f2_mul(t[0], w); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[4]; ang[0] = f2_fma(t[2], w, ang[0]); v[2] = f2_mul(y[0], w); } \
      { const f2 w = rows[5]; ang[1] = f2_mul(t[0], w); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[6]; ang[1] = f2_fma(t[1], w, ang[1]); v[1] = f2_mul(y[1], w); } \
      { const f2 w = rows[7]; ang[2] = f2_mul(t[0], w); v[0] = f2_fma(y[2], w, v[0]); } \
      ROWS(3) { const f2 w = rows[0]; ang[2] = f2_fma(t[1], w, ang[2]); v[1] = f2_fma(y[2], w, v[1]); } \
      { const f2 w = rows[1]; ang[2] = f2_fma(t[2], w, ang[2]); v[2] = f2_fma(y[2], w, v[2]); } \
      { const f2 w = rows[2]; ang[3] = f2_mul(t[1], w); v[1] = f2_fma(y[3], w, v[1]); } \
      { const f2 w = rows[3]; ang[3] = f2_fma(t[2], w, ang[3]); v[2] = f2_fma(y[3], w, v[2]); } \
      { const f2 w = rows[4]; ang[4] = f2_mul(t[0], w); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[5]; ang[4] = f2_fma(t[2], w, ang[4]); v[2] = f2_fma(y[4], w, v[2]); } \
      hadj[1] = f2_fma(R, v[0], hadj[1]); yw = f2_mul(h[1], v[0]); \
      hadj[2] = f2_fma(R, v[1], hadj[2]); yw = f2_fma(h[2], v[1], yw); \
      hadj[3] = f2_fma(R, v[2], hadj[3]); yw = f2_fma(h[3], v[2], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 5: edge l=2, source l=0 -> l=2 */ RADIAL(5) f2 yw, t[1], v[1]; \
      t[0] = f2_mul(R, h[0]); \
      { const f2 w = rows[6]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[7]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      ROWS(4) { const f2 w = rows[0]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      { const f2 w = rows[1]; ang[3] = f2_fma(t[0], w, ang[3]); v[0] = f2_fma(y[3], w, v[0]); } \
      { const f2 w = rows[2]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      hadj[0] = f2_fma(R, v[0], hadj[0]); yw = f2_mul(h[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 9: edge l=2, source l=1 -> l=3 */ RADIAL(9) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, h[1]); \
      t[1] = f2_mul(R, h[2]); \
      t[2] = f2_mul(R, h[3]); \
      { const f2 w = rows[3]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[4]; ang[0] = f2_fma(t[1], w, ang[0]); v[1] = f2_mul(y[0], w); } \
      { const f2 w = rows[5]; ang[0] = f2_fma(t[2], w, ang[0]); v[2] = f2_mul(y[0], w); } \
      { const f2 w = rows[6]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[7]; ang[1] = f2_fma(t[1], w, ang[1]); v[1] = f2_fma(y[1], w, v[1]); } \
      ROWS(5) { const f2 w = rows[0]; ang[1] = f2_fma(t[2], w, ang[1]); v[2] = f2_fma(y[1], w, v[2]); } \
      { const f2 w = rows[1]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      { const f2 w = rows[2]; ang[2] = f2_fma(t[1], w, ang[2]); v[1] = f2_fma(y[2], w, v[1]); } \
      { const f2 w = rows[3]; ang[2] = f2_fma(t[2], w, ang[2]); v[2] = f2_fma(y[2], w, v[2]); } \
      { const f2 w = rows[4]; ang[3] = f2_fma(t[0], w, ang[3]); v[0] = f2_fma(y[3], w, v[0]); } \
      { const f2 w = rows[5]; ang[3] = f2_fma(t[1], w, ang[3]); v[1] = f2_fma(y[3], w, v[1]); } \
      { const f2 w = rows[6]; ang[3] = f2_fma(t[2], w, ang[3]); v[2] = f2_fma(y[3], w, v[2]); } \
      { const f2 w = rows[7]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      ROWS(6) { const f2 w = rows[0]; ang[4] = f2_fma(t[1], w, ang[4]); v[1] = f2_fma(y[4], w, v[1]); } \
      { const f2 w = rows[1]; ang[4] = f2_fma(t[2], w, ang[4]); v[2] = f2_fma(y[4], w, v[2]); } \
      hadj[1] = f2_fma(R, v[0], hadj[1]); yw = f2_mul(h[1], v[0]); \
      hadj[2] = f2_fma(R, v[1], hadj[2]); yw = f2_fma(h[2], v[1], yw); \
      hadj[3] = f2_fma(R, v[2], hadj[3]); yw = f2_fma(h[3], v[2], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
      f[4] = f2_sum(ang[0]); f[5] = f2_sum(ang[1]); f[6] = f2_sum(ang[2]); f[7] = f2_sum(ang[3]); f[8] = f2_sum(ang[4]); \
    } \
    { f2 y[7], ang[7]; load_pair_harmonics<3>(yrow, y); \
    { /* path 7: edge l=3, source l=1 -> l=2 */ RADIAL(7) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, h[1]); \
      t[1] = f2_mul(R, h[2]); \
      t[2] = f2_mul(R, h[3]); \
      { const f2 w = rows[2]; ang[0] = f2_mul(t[0], w); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[3]; ang[0] = f2_fma(t[2], w, ang[0]); v[2] = f2_mul(y[0], w); } \
      { const f2 w = rows[4]; ang[1] = f2_mul(t[0], w); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[5]; ang[1] = f2_fma(t[1], w, ang[1]); v[1] = f2_mul(y[1], w); } \
      { const f2 w = rows[6]; ang[1] = f2_fma(t[2], w, ang[1]); v[2] = f2_fma(y[1], w, v[2]); } \
      { const f2 w = rows[7]; ang[2] = f2_mul(t[0], w); v[0] = f2_fma(y[2], w, v[0]); } \
      ROWS(7) { const f2 w = rows[0]; ang[2] = f2_fma(t[1], w, ang[2]); v[1] = f2_fma(y[2], w, v[1]); } \
      { const f2 w = rows[1]; ang[2] = f2_fma(t[2], w, ang[2]); v[2] = f2_fma(y[2], w, v[2]); } \
      { const f2 w = rows[2]; ang[3] = f2_mul(t[0], w); v[0] = f2_fma(y[3], w, v[0]); } \
      { const f2 w = rows[3]; ang[3] = f2_fma(t[1], w, ang[3]); v[1] = f2_fma(y[3], w, v[1]); } \
      { const f2 w = rows[4]; ang[3] = f2_fma(t[2], w, ang[3]); v[2] = f2_fma(y[3], w, v[2]); } \
      { const f2 w = rows[5]; ang[4] = f2_mul(t[0], w); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[6]; ang[4] = f2_fma(t[1], w, ang[4]); v[1] = f2_fma(y[4], w, v[1]); } \
      { const f2 w = rows[7]; ang[4] = f2_fma(t[2], w, ang[4]); v[2] = f2_fma(y[4], w, v[2]); } \
      ROWS(8) { const f2 w = rows[0]; ang[5] = f2_mul(t[0], w); v[0] = f2_fma(y[5], w, v[0]); } \
      { const f2 w = rows[1]; ang[5] = f2_fma(t[1], w, ang[5]); v[1] = f2_fma(y[5], w, v[1]); } \
      { const f2 w = rows[2]; ang[5] = f2_fma(t[2], w, ang[5]); v[2] = f2_fma(y[5], w, v[2]); } \
      { const f2 w = rows[3]; ang[6] = f2_mul(t[0], w); v[0] = f2_fma(y[6], w, v[0]); } \
      { const f2 w = rows[4]; ang[6] = f2_fma(t[2], w, ang[6]); v[2] = f2_fma(y[6], w, v[2]); } \
      hadj[1] = f2_fma(R, v[0], hadj[1]); yw = f2_mul(h[1], v[0]); \
      hadj[2] = f2_fma(R, v[1], hadj[2]); yw = f2_fma(h[2], v[1], yw); \
      hadj[3] = f2_fma(R, v[2], hadj[3]); yw = f2_fma(h[3], v[2], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 8: edge l=3, source l=0 -> l=3 */ RADIAL(8) f2 yw, t[1], v[1]; \
      t[0] = f2_mul(R, h[0]); \
      { const f2 w = rows[5]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[6]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[7]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      ROWS(9) { const f2 w = rows[0]; ang[3] = f2_fma(t[0], w, ang[3]); v[0] = f2_fma(y[3], w, v[0]); } \
      { const f2 w = rows[1]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[2]; ang[5] = f2_fma(t[0], w, ang[5]); v[0] = f2_fma(y[5], w, v[0]); } \
      { const f2 w = rows[3]; ang[6] = f2_fma(t[0], w, ang[6]); v[0] = f2_fma(y[6], w, v[0]); } \
      hadj[0] = f2_fma(R, v[0], hadj[0]); yw = f2_mul(h[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
      f[9] = f2_sum(ang[0]); f[10] = f2_sum(ang[1]); f[11] = f2_sum(ang[2]); f[12] = f2_sum(ang[3]); f[13] = f2_sum(ang[4]); f[14] = f2_sum(ang[5]); f[15] = f2_sum(ang[6]); \
    }
#define SXB_S1_L1_ADJOINT_ROWS \
    TERM(0, 0, 0) \
    TERM(1, 1, 3) \
    TERM(2, 2, 6) \
    TERM(3, 3, 9) \
    TERM(4, 5, 1) \
    TERM(5, 12, 1) \
    TERM(6, 18, 1) \
    TERM(7, 4, 2) STORE(0) \
    TERM(0, 10, 5) \
    TERM(1, 15, 8) \
    TERM(2, 6, 18) TERM_ADD(2, 7, 24) \
    TERM(3, 8, 15) \
    TERM(4, 9, 12) \
    TERM(5, 11, 15) \
    TERM(6, 13, 18) \
    TERM(7, 14, 21) STORE(1) \
    TERM(0, 16, 12) \
    TERM(1, 17, 21) \
    TERM(2, 19, 18) TERM_ADD(2, 20, 24) \
    TERM(3, 22, 10) \
    TERM(4, 26, 4) \
    TERM(5, 30, 7) \
    TERM(6, 33, 4) \
    TERM(7, 37, 4) STORE(2) \
    TERM(0, 39, 7) \
    TERM(1, 41, 10) \
    TERM(2, 45, 10) \
    TERM(3, 47, 7) \
    TERM(4, 51, 4) \
    TERM(5, 55, 10) \
    TERM(6, 21, 11) \
    TERM(7, 29, 14) STORE(3) \
    TERM(0, 36, 17) \
    TERM(1, 43, 20) \
    TERM(2, 50, 23) \
    TERM(3, 23, 35) TERM_ADD(3, 24, 39) \
    TERM(4, 25, 29) \
    TERM(5, 27, 27) TERM_ADD(5, 28, 31) \
    TERM(6, 31, 33) TERM_ADD(6, 32, 37) \
    TERM(7, 34, 31) STORE(4) \
    TERM(0, 35, 29) \
    TERM(1, 38, 31) \
    TERM(2, 40, 33) \
    TERM(3, 42, 35) \
    TERM(4, 44, 29) \
    TERM(5, 46, 35) \
    TERM(6, 48, 33) TERM_ADD(6, 49, 37) \
    TERM(7, 52, 27) TERM_ADD(7, 53, 31) STORE(5) \
    TERM(0, 54, 37) \
    TERM(1, 56, 35) TERM_ADD(1, 57, 39) \
    TERM(2, 59, 25) \
    TERM(3, 60, 13) \
    TERM(4, 62, 22) \
    TERM(5, 63, 13) \
    TERM(6, 64, 16) \
    TERM(7, 66, 19) TERM_ADD(7, 67, 25) STORE(6) \
    TERM(0, 68, 16) \
    TERM(1, 69, 13) \
    TERM(2, 71, 16) \
    TERM(3, 72, 19) \
    TERM(4, 73, 22) \
    TERM(5, 75, 13) \
    TERM(6, 76, 22) \
    TERM(7, 77, 19) TERM_ADD(7, 78, 25) STORE(7) \
    TERM(0, 80, 16) \
    TERM(1, 81, 25) \
    TERM(2, 82, 22) \
    TERM(3, 84, 13) \
    TERM(4, 85, 25) \
    TERM(5, 58, 26) \
    TERM(6, 61, 28) \
    TERM(7, 65, 30) STORE(8) \
    TERM(0, 70, 32) \
    TERM(1, 74, 34) \
    TERM(2, 79, 36) \
    TERM(3, 83, 38) \
    v[4] = 0ull; \
    v[5] = 0ull; \
    v[6] = 0ull; \
    v[7] = 0ull; STORE(9)

// ---- shape S2: edge l_max=3, hidden L_max=2
#define SXB_S2_LMAX 3
#define SXB_S2_HIDDEN_LMAX 2
#define SXB_S2_NUM_LM 16
#define SXB_S2_NUM_HIDDEN 9
#define SXB_S2_NUM_PATHS 17
#define SXB_S2_NUM_ROWS 243
#define SXB_S2_NUM_LME 71
#define SXB_S2_NUM_TERMS 215
// X(path, l_out, l_edge, l_source, first_row)
#define SXB_S2_PATHS(X) \
    X(0, 0, 0, 0, 0) \
    X(1, 0, 1, 1, 1) \
    X(2, 0, 2, 2, 10) \
    X(3, 1, 1, 0, 35) \
    X(4, 1, 0, 1, 38) \
    X(5, 1, 2, 1, 41) \
    X(6, 1, 1, 2, 56) \
    X(7, 1, 3, 2, 71) \
    X(8, 2, 2, 0, 106) \
    X(9, 2, 1, 1, 111) \
    X(10, 2, 3, 1, 120) \
    X(11, 2, 0, 2, 141) \
    X(12, 2, 2, 2, 146) \
    X(13, 3, 3, 0, 171) \
    X(14, 3, 2, 1, 178) \
    X(15, 3, 1, 2, 193) \
    X(16, 3, 3, 2, 208)
// X(row, path, lm_edge, lm_source)
#define SXB_S2_ROWS(X) \
    X(0, 0, 0, 0) \
    X(1, 1, 1, 1) \
    X(2, 1, 1, 2) \
    X(3, 1, 1, 3) \
    X(4, 1, 2, 1) \
    X(5, 1, 2, 2) \
    X(6, 1, 2, 3) \
    X(7, 1, 3, 1) \
    X(8, 1, 3, 2) \
    X(9, 1, 3, 3) \
    X(10, 2, 4, 4) \
    X(11, 2, 4, 5) \
    X(12, 2, 4, 6) \
    X(13, 2, 4, 7) \
    X(14, 2, 4, 8) \
    X(15, 2, 5, 4) \
    X(16, 2, 5, 5) \
    X(17, 2, 5, 6) \
    X(18, 2, 5, 7) \
    X(19, 2, 5, 8) \
    X(20, 2, 6, 4) \
    X(21, 2, 6, 5) \
    X(22, 2, 6, 6) \
    X(23, 2, 6, 7) \
    X(24, 2, 6, 8) \
    X(25, 2, 7, 4) \
    X(26, 2, 7, 5) \
    X(27, 2, 7, 6) \
    X(28, 2, 7, 7) \
    X(29, 2, 7, 8) \
    X(30, 2, 8, 4) \
    X(31, 2, 8, 5) \
    X(32, 2, 8, 6) \
    X(33, 2, 8, 7) \
    X(34, 2, 8, 8) \
    X(35, 3, 1, 0) \
    X(36, 3, 2, 0) \
    X(37, 3, 3, 0) \
    X(38, 4, 0, 1) \
    X(39, 4, 0, 2) \
    X(40, 4, 0, 3) \
    X(41, 5, 4, 1) \
    X(42, 5, 4, 2) \
    X(43, 5, 4, 3) \
    X(44, 5, 5, 1) \
    X(45, 5, 5, 2) \
    X(46, 5, 5, 3) \
    X(47, 5, 6, 1) \
    X(48, 5, 6, 2) \
    X(49, 5, 6, 3) \
    X(50, 5, 7, 1) \
    X(51, 5, 7, 2) \
    X(52, 5, 7, 3) \
    X(53, 5, 8, 1) \
    X(54, 5, 8, 2) \
    X(55, 5, 8, 3) \
    X(56, 6, 1, 4) \
    X(57, 6, 1, 5) \
    X(58, 6, 1, 6) \
    X(59, 6, 1, 7) \
    X(60, 6, 1, 8) \
    X(61, 6, 2, 4) \
    X(62, 6, 2, 5) \
    X(63, 6, 2, 6) \
    X(64, 6, 2, 7) \
    X(65, 6, 2, 8) \
    X(66, 6, 3, 4) \
    X(67, 6, 3, 5) \
    X(68, 6, 3, 6) \
    X(69, 6, 3, 7) \
    X(70, 6, 3, 8) \
    X(71, 7, 9, 4) \
    X(72, 7, 9, 5) \
    X(73, 7, 9, 6) \
    X(74, 7, 9, 7) \
    X(75, 7, 9, 8) \
    X(76, 7, 10, 4) \
    X(77, 7, 10, 5) \
    X(78, 7, 10, 6) \
    X(79, 7, 10, 7) \
    X(80, 7, 10, 8) \
    X(81, 7, 11, 4) \
    X(82, 7, 11, 5) \
    X(83, 7, 11, 6) \
    X(84, 7, 11, 7) \
    X(85, 7, 11, 8) \
    X(86, 7, 12, 4) \
    X(87, 7, 12, 5) \
    X(88, 7, 12, 6) \
    X(89, 7, 12, 7) \
    X(90, 7, 12, 8) \
    X(91, 7, 13, 4) \
    X(92, 7, 13, 5) \
    X(93, 7, 13, 6) \
    X(94, 7, 13, 7) \
    X(95, 7, 13, 8) \
    X(96, 7, 14, 4) \
    X(97, 7, 14, 5) \
    X(98, 7, 14, 6) \
    X(99, 7, 14, 7) \
    X(100, 7, 14, 8) \
    X(101, 7, 15, 4) \
    X(102, 7, 15, 5) \
    X(103, 7, 15, 6) \
    X(104, 7, 15, 7) \
    X(105, 7, 15, 8) \
    X(106, 8, 4, 0) \
    X(107, 8, 5, 0) \
    X(108, 8, 6, 0) \
    X(109, 8, 7, 0) \
    X(110, 8, 8, 0) \
    X(111, 9, 1, 1) \
    X(112, 9, 1, 2) \
    X(113, 9, 1, 3) \
    X(114, 9, 2, 1) \
    X(115, 9, 2, 2) \
    X(116, 9, 2, 3) \
    X(117, 9, 3, 1) \
    X(118, 9, 3, 2) \
    X(119, 9, 3, 3) \
    X(120, 10, 9, 1) \
    X(121, 10, 9, 2) \
    X(122, 10, 9, 3) \
    X(123, 10, 10, 1) \
    X(124, 10, 10, 2) \
    X(125, 10, 10, 3) \
    X(126, 10, 11, 1) \
    X(127, 10, 11, 2) \
    X(128, 10, 11, 3) \
    X(129, 10, 12, 1) \
    X(130, 10, 12, 2) \
    X(131, 10, 12, 3) \
    X(132, 10, 13, 1) \
    X(133, 10, 13, 2) \
    X(134, 10, 13, 3) \
    X(135, 10, 14, 1) \
    X(136, 10, 14, 2) \
    X(137, 10, 14, 3) \
    X(138, 10, 15, 1) \
    X(139, 10, 15, 2) \
    X(140, 10, 15, 3) \
    X(141, 11, 0, 4) \
    X(142, 11, 0, 5) \
    X(143, 11, 0, 6) \
    X(144, 11, 0, 7) \
    X(145, 11, 0, 8) \
    X(146, 12, 4, 4) \
    X(147, 12, 4, 5) \
    X(148, 12, 4, 6) \
    X(149, 12, 4, 7) \
    X(150, 12, 4, 8) \
    X(151, 12, 5, 4) \
    X(152, 12, 5, 5) \
    X(153, 12, 5, 6) \
    X(154, 12, 5, 7) \
    X(155, 12, 5, 8) \
    X(156, 12, 6, 4) \
    X(157, 12, 6, 5) \
    X(158, 12, 6, 6) \
    X(159, 12, 6, 7) \
    X(160, 12, 6, 8) \
    X(161, 12, 7, 4) \
    X(162, 12, 7, 5) \
    X(163, 12, 7, 6) \
    X(164, 12, 7, 7) \
    X(165, 12, 7, 8) \
    X(166, 12, 8, 4) \
    X(167, 12, 8, 5) \
    X(168, 12, 8, 6) \
    X(169, 12, 8, 7) \
    X(170, 12, 8, 8) \
    X(171, 13, 9, 0) \
    X(172, 13, 10, 0) \
    X(173, 13, 11, 0) \
    X(174, 13, 12, 0) \
    X(175, 13, 13, 0) \
    X(176, 13, 14, 0) \
    X(177, 13, 15, 0) \
    X(178, 14, 4, 1) \
    X(179, 14, 4, 2) \
    X(180, 14, 4, 3) \
    X(181, 14, 5, 1) \
    X(182, 14, 5, 2) \
    X(183, 14, 5, 3) \
    X(184, 14, 6, 1) \
    X(185, 14, 6, 2) \
    X(186, 14, 6, 3) \
    X(187, 14, 7, 1) \
    X(188, 14, 7, 2) \
    X(189, 14, 7, 3) \
    X(190, 14, 8, 1) \
    X(191, 14, 8, 2) \
    X(192, 14, 8, 3) \
    X(193, 15, 1, 4) \
    X(194, 15, 1, 5) \
    X(195, 15, 1, 6) \
    X(196, 15, 1, 7) \
    X(197, 15, 1, 8) \
    X(198, 15, 2, 4) \
    X(199, 15, 2, 5) \
    X(200, 15, 2, 6) \
    X(201, 15, 2, 7) \
    X(202, 15, 2, 8) \
    X(203, 15, 3, 4) \
    X(204, 15, 3, 5) \
    X(205, 15, 3, 6) \
    X(206, 15, 3, 7) \
    X(207, 15, 3, 8) \
    X(208, 16, 9, 4) \
    X(209, 16, 9, 5) \
    X(210, 16, 9, 6) \
    X(211, 16, 9, 7) \
    X(212, 16, 9, 8) \
    X(213, 16, 10, 4) \
    X(214, 16, 10, 5) \
    X(215, 16, 10, 6) \
    X(216, 16, 10, 7) \
    X(217, 16, 10, 8) \
    X(218, 16, 11, 4) \
    X(219, 16, 11, 5) \
    X(220, 16, 11, 6) \
    X(221, 16, 11, 7) \
    X(222, 16, 11, 8) \
    X(223, 16, 12, 4) \
    X(224, 16, 12, 5) \
    X(225, 16, 12, 6) \
    X(226, 16, 12, 7) \
    X(227, 16, 12, 8) \
    X(228, 16, 13, 4) \
    X(229, 16, 13, 5) \
    X(230, 16, 13, 6) \
    X(231, 16, 13, 7) \
    X(232, 16, 13, 8) \
    X(233, 16, 14, 4) \
    X(234, 16, 14, 5) \
    X(235, 16, 14, 6) \
    X(236, 16, 14, 7) \
    X(237, 16, 14, 8) \
    X(238, 16, 15, 4) \
    X(239, 16, 15, 5) \
    X(240, 16, 15, 6) \
    X(241, 16, 15, 7) \
    X(242, 16, 15, 8)
// X(term, row, lme): coefficient values live in constant memory, indexed by term
#define SXB_S2_TERMS(X) \
    X(0, 0, 0) \
    X(1, 38, 4) \
    X(2, 39, 9) \
    X(3, 40, 14) \
    X(4, 141, 21) \
    X(5, 142, 26) \
    X(6, 143, 31) \
    X(7, 144, 36) \
    X(8, 145, 41) \
    X(9, 35, 3) \
    X(10, 1, 1) \
    X(11, 111, 29) \
    X(12, 111, 39) \
    X(13, 112, 24) \
    X(14, 113, 19) \
    X(15, 56, 16) \
    X(16, 193, 61) \
    X(17, 193, 69) \
    X(18, 57, 11) \
    X(19, 194, 57) \
    X(20, 194, 65) \
    X(21, 58, 6) \
    X(22, 195, 53) \
    X(23, 196, 49) \
    X(24, 60, 6) \
    X(25, 197, 45) \
    X(26, 197, 53) \
    X(27, 36, 8) \
    X(28, 114, 24) \
    X(29, 5, 1) \
    X(30, 115, 29) \
    X(31, 116, 34) \
    X(32, 198, 49) \
    X(33, 62, 6) \
    X(34, 199, 53) \
    X(35, 63, 11) \
    X(36, 200, 57) \
    X(37, 64, 16) \
    X(38, 201, 61) \
    X(39, 202, 65) \
    X(40, 37, 13) \
    X(41, 117, 19) \
    X(42, 118, 34) \
    X(43, 9, 1) \
    X(44, 119, 29) \
    X(45, 119, 39) \
    X(46, 66, 6) \
    X(47, 203, 45) \
    X(48, 203, 53) \
    X(49, 204, 49) \
    X(50, 68, 16) \
    X(51, 205, 61) \
    X(52, 69, 11) \
    X(53, 206, 57) \
    X(54, 206, 65) \
    X(55, 70, 16) \
    X(56, 207, 61) \
    X(57, 207, 69) \
    X(58, 106, 18) \
    X(59, 41, 15) \
    X(60, 178, 60) \
    X(61, 178, 68) \
    X(62, 179, 48) \
    X(63, 43, 5) \
    X(64, 180, 44) \
    X(65, 180, 52) \
    X(66, 10, 2) \
    X(67, 146, 32) \
    X(68, 147, 37) \
    X(69, 148, 22) \
    X(70, 149, 27) \
    X(71, 107, 23) \
    X(72, 44, 10) \
    X(73, 181, 56) \
    X(74, 181, 64) \
    X(75, 45, 5) \
    X(76, 182, 52) \
    X(77, 183, 48) \
    X(78, 151, 37) \
    X(79, 16, 2) \
    X(80, 152, 32) \
    X(81, 152, 42) \
    X(82, 153, 27) \
    X(83, 154, 22) \
    X(84, 155, 27) \
    X(85, 108, 28) \
    X(86, 47, 5) \
    X(87, 184, 52) \
    X(88, 48, 10) \
    X(89, 185, 56) \
    X(90, 49, 15) \
    X(91, 186, 60) \
    X(92, 156, 22) \
    X(93, 157, 27) \
    X(94, 22, 2) \
    X(95, 158, 32) \
    X(96, 159, 37) \
    X(97, 160, 42) \
    X(98, 109, 33) \
    X(99, 187, 48) \
    X(100, 51, 15) \
    X(101, 188, 60) \
    X(102, 52, 10) \
    X(103, 189, 56) \
    X(104, 189, 64) \
    X(105, 161, 27) \
    X(106, 162, 22) \
    X(107, 163, 37) \
    X(108, 28, 2) \
    X(109, 164, 32) \
    X(110, 164, 42) \
    X(111, 165, 37) \
    X(112, 110, 38) \
    X(113, 53, 5) \
    X(114, 190, 44) \
    X(115, 190, 52) \
    X(116, 191, 64) \
    X(117, 55, 15) \
    X(118, 192, 60) \
    X(119, 192, 68) \
    X(120, 167, 27) \
    X(121, 168, 42) \
    X(122, 169, 37) \
    X(123, 34, 2) \
    X(124, 170, 32) \
    X(125, 171, 43) \
    X(126, 120, 40) \
    X(127, 122, 20) \
    X(128, 71, 17) \
    X(129, 208, 62) \
    X(130, 209, 66) \
    X(131, 210, 46) \
    X(132, 211, 50) \
    X(133, 75, 7) \
    X(134, 212, 54) \
    X(135, 172, 47) \
    X(136, 123, 35) \
    X(137, 124, 20) \
    X(138, 125, 25) \
    X(139, 76, 12) \
    X(140, 213, 58) \
    X(141, 77, 17) \
    X(142, 214, 62) \
    X(143, 214, 70) \
    X(144, 79, 7) \
    X(145, 216, 46) \
    X(146, 216, 54) \
    X(147, 173, 51) \
    X(148, 126, 30) \
    X(149, 126, 40) \
    X(150, 127, 25) \
    X(151, 128, 20) \
    X(152, 81, 17) \
    X(153, 218, 62) \
    X(154, 218, 70) \
    X(155, 82, 12) \
    X(156, 219, 58) \
    X(157, 219, 66) \
    X(158, 83, 7) \
    X(159, 220, 54) \
    X(160, 221, 50) \
    X(161, 85, 7) \
    X(162, 222, 46) \
    X(163, 222, 54) \
    X(164, 174, 55) \
    X(165, 129, 25) \
    X(166, 130, 30) \
    X(167, 131, 35) \
    X(168, 223, 50) \
    X(169, 87, 7) \
    X(170, 224, 54) \
    X(171, 88, 12) \
    X(172, 225, 58) \
    X(173, 89, 17) \
    X(174, 226, 62) \
    X(175, 227, 66) \
    X(176, 175, 59) \
    X(177, 132, 20) \
    X(178, 133, 35) \
    X(179, 134, 30) \
    X(180, 134, 40) \
    X(181, 91, 7) \
    X(182, 228, 46) \
    X(183, 228, 54) \
    X(184, 229, 50) \
    X(185, 93, 17) \
    X(186, 230, 62) \
    X(187, 94, 12) \
    X(188, 231, 58) \
    X(189, 231, 66) \
    X(190, 95, 17) \
    X(191, 232, 62) \
    X(192, 232, 70) \
    X(193, 176, 63) \
    X(194, 135, 25) \
    X(195, 136, 40) \
    X(196, 137, 35) \
    X(197, 97, 7) \
    X(198, 234, 46) \
    X(199, 234, 54) \
    X(200, 99, 17) \
    X(201, 236, 62) \
    X(202, 236, 70) \
    X(203, 100, 12) \
    X(204, 237, 58) \
    X(205, 177, 67) \
    X(206, 138, 20) \
    X(207, 140, 40) \
    X(208, 101, 7) \
    X(209, 238, 54) \
    X(210, 239, 50) \
    X(211, 240, 70) \
    X(212, 241, 66) \
    X(213, 105, 17) \
    X(214, 242, 62)
// this library's own derivation of the coupling coefficients, by term (a model file carries its own)
#define SXB_S2_DEFAULT_CG {1.0f, 1.0f, 0.9999999999999998f, 1.0f, 1.0f, 1.0000000000000002f, 1.0000000000000007f, 1.0000000000000013f, 1.000000000000001f, 1.0f, 0.5773502691896257f, 0.40824829046386385f, 0.7071067811865485f, -0.7071067811865476f, -0.7071067811865471f, 0.547722557505166f, 0.1825741858350552f, 0.7071067811865475f, 0.547722557505166f, 0.44721359549995815f, 0.5773502691896256f, -0.31622776601683805f, -0.6324555320336767f, -0.5773502691896262f, -0.5477225575051661f, -0.7071067811865479f, -0.18257418583505508f, 0.9999999999999997f, -0.7071067811865471f, 0.5773502691896257f, -0.816496580927727f, -0.7071067811865479f, -0.5773502691896261f, 0.5477225575051663f, -0.730296743340222f, 0.6324555320336764f, -0.7745966692414837f, 0.547722557505166f, -0.7302967433402215f, -0.5773502691896262f, 0.9999999999999994f, -0.7071067811865478f, -0.7071067811865476f, 0.5773502691896258f, 0.4082482904638637f, -0.7071067811865486f, 0.5477225575051657f, -0.7071067811865474f, 0.1825741858350554f, -0.5773502691896262f, -0.3162277660168378f, -0.6324555320336757f, 0.5477225575051656f, 0.4472135954999579f, -0.5773502691896257f, 0.5477225575051661f, 0.18257418583505572f, -0.707106781186548f, 1.0f, 0.5477225575051663f, 0.1825741858350547f, 0.7071067811865475f, -0.5773502691896257f, 0.547722557505166f, -0.7071067811865475f, 0.18257418583505564f, 0.4472135954999578f, 0.534522483824848f, -0.4629100498862763f, 0.5345224838248486f, -0.4629100498862764f, 1.0000000000000004f, 0.5477225575051659f, 0.4472135954999578f, 0.577350269189626f, 0.547722557505166f, -0.7302967433402211f, -0.5773502691896253f, -0.4629100498862749f, 0.44721359549995787f, -0.26726124191242434f, 0.4629100498862759f, -0.2672612419124245f, -0.46291004988627593f, 0.4629100498862758f, 1.0000000000000013f, -0.3162277660168377f, -0.6324555320336763f, 0.6324555320336757f, -0.7745966692414836f, -0.31622776601683755f, -0.6324555320336758f, 0.5345224838248483f, -0.26726124191242423f, 0.44721359549995826f, -0.5345224838248486f, -0.26726124191242473f, 0.5345224838248492f, 1.0000000000000009f, -0.5773502691896265f, 0.547722557505166f, -0.7302967433402215f, 0.5477225575051659f, 0.4472135954999579f, -0.5773502691896257f, -0.46291004988627593f, -0.46291004988627615f, -0.2672612419124245f, 0.44721359549995787f, -0.2672612419124245f, -0.4629100498862757f, -0.4629100498862757f, 1.0000000000000013f, -0.5477225575051666f, -0.7071067811865475f, -0.1825741858350553f, -0.5773502691896262f, 0.547722557505166f, 0.18257418583505564f, -0.7071067811865474f, 0.4629100498862758f, 0.5345224838248491f, -0.46291004988627604f, 0.44721359549995826f, 0.5345224838248492f, 1.0f, 0.5976143046671968f, 0.5976143046671969f, 0.4629100498862755f, 0.28867513459481275f, -0.4564354645876392f, 0.6454972243679029f, -0.45643546458763806f, 0.4629100498862761f, 0.28867513459481325f, 1.0000000000000002f, 0.48795003647426666f, 0.4879500364742665f, 0.48795003647426605f, 0.37796447300922703f, 0.5773502691896255f, 0.3779644730092266f, -0.3535533905932735f, 0.45643546458763773f, 0.37796447300922714f, -0.45643546458763856f, -0.3535533905932737f, 1.0000000000000013f, 0.5345224838248491f, 0.1543033499620919f, 0.6172133998483681f, -0.15430334996209205f, -0.11952286093343935f, -0.4472135954999578f, -0.2886751345948131f, 0.4780914437337578f, -0.18257418583505527f, 0.35355339059327373f, 0.4140393356054125f, -0.38729833462074176f, -0.3535533905932738f, 0.11952286093343935f, 0.2886751345948131f, 0.4472135954999586f, 0.9999999999999994f, -0.3779644730092276f, 0.6546536707079776f, -0.37796447300922775f, 0.5773502691896262f, -0.29277002188456f, -0.1825741858350554f, 0.5070925528371099f, -0.5163977794943228f, -0.2927700218845599f, -0.1825741858350554f, 0.5773502691896263f, 0.999999999999999f, -0.15430334996209197f, 0.6172133998483679f, 0.5345224838248491f, -0.15430334996209194f, -0.11952286093343921f, 0.28867513459481287f, -0.4472135954999578f, -0.35355339059327345f, 0.4140393356054125f, -0.3872983346207412f, 0.4780914437337571f, -0.1825741858350554f, -0.3535533905932738f, -0.1195228609334394f, -0.44721359549995787f, 0.2886751345948128f, 0.9999999999999997f, -0.48795003647426655f, 0.4879500364742668f, 0.4879500364742665f, -0.37796447300922714f, -0.4564354645876383f, 0.3535533905932735f, 0.37796447300922686f, -0.3535533905932738f, -0.4564354645876384f, 0.3779644730092276f, 0.5773502691896266f, 1.0000000000000002f, -0.5976143046671967f, 0.5976143046671976f, -0.4629100498862756f, -0.28867513459481287f, 0.45643546458763795f, 0.645497224367903f, -0.4564354645876388f, 0.46291004988627577f, 0.2886751345948131f}
#define SXB_S2_M0_NUM_TERMS 887
#define SXB_S2_M0_OFFSETS {0, 94, 206, 298, 410, 500, 597, 692, 789, 887}
// X1(out, term, a)  X2(out, term, a, b)  X3(out, term, a, b, c)
#define SXB_S2_M0_TERMS(X1, X2, X3) \
    X1(0, 0, 0) \
    X1(1, 94, 1) \
    X1(2, 206, 2) \
    X1(3, 298, 3) \
    X1(4, 410, 4) \
    X1(5, 500, 5) \
    X1(6, 597, 6) \
    X1(7, 692, 7) \
    X1(8, 789, 8) \
    X2(0, 1, 0, 0) \
    X2(0, 2, 1, 1) \
    X2(0, 3, 2, 2) \
    X2(0, 4, 3, 3) \
    X2(0, 5, 4, 4) \
    X2(0, 6, 5, 5) \
    X2(0, 7, 6, 6) \
    X2(0, 8, 7, 7) \
    X2(0, 9, 8, 8) \
    X2(0, 10, 9, 9) \
    X2(0, 11, 10, 10) \
    X2(0, 12, 11, 11) \
    X2(0, 13, 12, 12) \
    X2(0, 14, 13, 13) \
    X2(0, 15, 14, 14) \
    X2(0, 16, 15, 15) \
    X2(1, 95, 0, 1) \
    X2(1, 96, 1, 6) \
    X2(1, 97, 1, 8) \
    X2(1, 98, 2, 5) \
    X2(1, 99, 3, 4) \
    X2(1, 100, 4, 13) \
    X2(1, 101, 4, 15) \
    X2(1, 102, 5, 12) \
    X2(1, 103, 5, 14) \
    X2(1, 104, 6, 11) \
    X2(1, 105, 7, 10) \
    X2(1, 106, 8, 9) \
    X2(1, 107, 8, 11) \
    X2(2, 207, 0, 2) \
    X2(2, 208, 1, 5) \
    X2(2, 209, 2, 6) \
    X2(2, 210, 3, 7) \
    X2(2, 211, 4, 10) \
    X2(2, 212, 5, 11) \
    X2(2, 213, 6, 12) \
    X2(2, 214, 7, 13) \
    X2(2, 215, 8, 14) \
    X2(3, 299, 0, 3) \
    X2(3, 300, 1, 4) \
    X2(3, 301, 2, 7) \
    X2(3, 302, 3, 6) \
    X2(3, 303, 3, 8) \
    X2(3, 304, 4, 9) \
    X2(3, 305, 4, 11) \
    X2(3, 306, 5, 10) \
    X2(3, 307, 6, 13) \
    X2(3, 308, 7, 12) \
    X2(3, 309, 7, 14) \
    X2(3, 310, 8, 13) \
    X2(3, 311, 8, 15) \
    X2(4, 411, 0, 4) \
    X2(4, 412, 1, 3) \
    X2(4, 413, 1, 13) \
    X2(4, 414, 1, 15) \
    X2(4, 415, 2, 10) \
    X2(4, 416, 3, 9) \
    X2(4, 417, 3, 11) \
    X2(4, 418, 4, 6) \
    X2(4, 419, 5, 7) \
    X2(4, 420, 9, 13) \
    X2(4, 421, 10, 12) \
    X2(4, 422, 11, 13) \
    X2(4, 423, 11, 15) \
    X2(5, 501, 0, 5) \
    X2(5, 502, 1, 2) \
    X2(5, 503, 1, 12) \
    X2(5, 504, 1, 14) \
    X2(5, 505, 2, 11) \
    X2(5, 506, 3, 10) \
    X2(5, 507, 4, 7) \
    X2(5, 508, 5, 6) \
    X2(5, 509, 5, 8) \
    X2(5, 510, 9, 14) \
    X2(5, 511, 10, 13) \
    X2(5, 512, 10, 15) \
    X2(5, 513, 11, 12) \
    X2(5, 514, 11, 14) \
    X2(6, 598, 0, 6) \
    X2(6, 599, 1, 1) \
    X2(6, 600, 1, 11) \
    X2(6, 601, 2, 2) \
    X2(6, 602, 2, 12) \
    X2(6, 603, 3, 3) \
    X2(6, 604, 3, 13) \
    X2(6, 605, 4, 4) \
    X2(6, 606, 5, 5) \
    X2(6, 607, 6, 6) \
    X2(6, 608, 7, 7) \
    X2(6, 609, 8, 8) \
    X2(6, 610, 9, 9) \
    X2(6, 611, 11, 11) \
    X2(6, 612, 12, 12) \
    X2(6, 613, 13, 13) \
    X2(6, 614, 15, 15) \
    X2(7, 693, 0, 7) \
    X2(7, 694, 1, 10) \
    X2(7, 695, 2, 3) \
    X2(7, 696, 2, 13) \
    X2(7, 697, 3, 12) \
    X2(7, 698, 3, 14) \
    X2(7, 699, 4, 5) \
    X2(7, 700, 6, 7) \
    X2(7, 701, 7, 8) \
    X2(7, 702, 9, 10) \
    X2(7, 703, 10, 11) \
    X2(7, 704, 12, 13) \
    X2(7, 705, 13, 14) \
    X2(7, 706, 14, 15) \
    X2(8, 790, 0, 8) \
    X2(8, 791, 1, 1) \
    X2(8, 792, 1, 9) \
    X2(8, 793, 1, 11) \
    X2(8, 794, 2, 14) \
    X2(8, 795, 3, 3) \
    X2(8, 796, 3, 13) \
    X2(8, 797, 3, 15) \
    X2(8, 798, 5, 5) \
    X2(8, 799, 6, 8) \
    X2(8, 800, 7, 7) \
    X2(8, 801, 9, 11) \
    X2(8, 802, 11, 11) \
    X2(8, 803, 12, 14) \
    X2(8, 804, 13, 13) \
    X2(8, 805, 13, 15) \
    X3(0, 17, 0, 0, 0) \
    X3(0, 18, 0, 1, 1) \
    X3(0, 19, 0, 2, 2) \
    X3(0, 20, 0, 3, 3) \
    X3(0, 21, 0, 4, 4) \
    X3(0, 22, 0, 5, 5) \
    X3(0, 23, 0, 6, 6) \
    X3(0, 24, 0, 7, 7) \
    X3(0, 25, 0, 8, 8) \
    X3(0, 26, 0, 9, 9) \
    X3(0, 27, 0, 10, 10) \
    X3(0, 28, 0, 11, 11) \
    X3(0, 29, 0, 12, 12) \
    X3(0, 30, 0, 13, 13) \
    X3(0, 31, 0, 14, 14) \
    X3(0, 32, 0, 15, 15) \
    X3(0, 33, 1, 1, 6) \
    X3(0, 34, 1, 1, 8) \
    X3(0, 35, 1, 2, 5) \
    X3(0, 36, 1, 3, 4) \
    X3(0, 37, 1, 4, 13) \
    X3(0, 38, 1, 4, 15) \
    X3(0, 39, 1, 5, 12) \
    X3(0, 40, 1, 5, 14) \
    X3(0, 41, 1, 6, 11) \
    X3(0, 42, 1, 7, 10) \
    X3(0, 43, 1, 8, 9) \
    X3(0, 44, 1, 8, 11) \
    X3(0, 45, 2, 2, 6) \
    X3(0, 46, 2, 3, 7) \
    X3(0, 47, 2, 4, 10) \
    X3(0, 48, 2, 5, 11) \
    X3(0, 49, 2, 6, 12) \
    X3(0, 50, 2, 7, 13) \
    X3(0, 51, 2, 8, 14) \
    X3(0, 52, 3, 3, 6) \
    X3(0, 53, 3, 3, 8) \
    X3(0, 54, 3, 4, 9) \
    X3(0, 55, 3, 4, 11) \
    X3(0, 56, 3, 5, 10) \
    X3(0, 57, 3, 6, 13) \
    X3(0, 58, 3, 7, 12) \
    X3(0, 59, 3, 7, 14) \
    X3(0, 60, 3, 8, 13) \
    X3(0, 61, 3, 8, 15) \
    X3(0, 62, 4, 4, 6) \
    X3(0, 63, 4, 5, 7) \
    X3(0, 64, 4, 9, 13) \
    X3(0, 65, 4, 10, 12) \
    X3(0, 66, 4, 11, 13) \
    X3(0, 67, 4, 11, 15) \
    X3(0, 68, 5, 5, 6) \
    X3(0, 69, 5, 5, 8) \
    X3(0, 70, 5, 9, 14) \
    X3(0, 71, 5, 10, 13) \
    X3(0, 72, 5, 10, 15) \
    X3(0, 73, 5, 11, 12) \
    X3(0, 74, 5, 11, 14) \
    X3(0, 75, 6, 6, 6) \
    X3(0, 76, 6, 7, 7) \
    X3(0, 77, 6, 8, 8) \
    X3(0, 78, 6, 9, 9) \
    X3(0, 79, 6, 11, 11) \
    X3(0, 80, 6, 12, 12) \
    X3(0, 81, 6, 13, 13) \
    X3(0, 82, 6, 15, 15) \
    X3(0, 83, 7, 7, 8) \
    X3(0, 84, 7, 9, 10) \
    X3(0, 85, 7, 10, 11) \
    X3(0, 86, 7, 12, 13) \
    X3(0, 87, 7, 13, 14) \
    X3(0, 88, 7, 14, 15) \
    X3(0, 89, 8, 9, 11) \
    X3(0, 90, 8, 11, 11) \
    X3(0, 91, 8, 12, 14) \
    X3(0, 92, 8, 13, 13) \
    X3(0, 93, 8, 13, 15) \
    X3(1, 108, 0, 0, 1) \
    X3(1, 109, 0, 1, 6) \
    X3(1, 110, 0, 1, 8) \
    X3(1, 111, 0, 2, 5) \
    X3(1, 112, 0, 3, 4) \
    X3(1, 113, 0, 4, 13) \
    X3(1, 114, 0, 4, 15) \
    X3(1, 115, 0, 5, 12) \
    X3(1, 116, 0, 5, 14) \
    X3(1, 117, 0, 6, 11) \
    X3(1, 118, 0, 7, 10) \
    X3(1, 119, 0, 8, 9) \
    X3(1, 120, 0, 8, 11) \
    X3(1, 121, 1, 1, 1) \
    X3(1, 122, 1, 1, 9) \
    X3(1, 123, 1, 1, 11) \
    X3(1, 124, 1, 2, 2) \
    X3(1, 125, 1, 2, 12) \
    X3(1, 126, 1, 2, 14) \
    X3(1, 127, 1, 3, 3) \
    X3(1, 128, 1, 3, 13) \
    X3(1, 129, 1, 3, 15) \
    X3(1, 130, 1, 4, 4) \
    X3(1, 131, 1, 5, 5) \
    X3(1, 132, 1, 6, 6) \
    X3(1, 133, 1, 6, 8) \
    X3(1, 134, 1, 7, 7) \
    X3(1, 135, 1, 8, 8) \
    X3(1, 136, 1, 9, 9) \
    X3(1, 137, 1, 9, 11) \
    X3(1, 138, 1, 10, 10) \
    X3(1, 139, 1, 11, 11) \
    X3(1, 140, 1, 12, 12) \
    X3(1, 141, 1, 12, 14) \
    X3(1, 142, 1, 13, 13) \
    X3(1, 143, 1, 13, 15) \
    X3(1, 144, 1, 14, 14) \
    X3(1, 145, 1, 15, 15) \
    X3(1, 146, 2, 2, 11) \
    X3(1, 147, 2, 3, 10) \
    X3(1, 148, 2, 4, 7) \
    X3(1, 149, 2, 5, 6) \
    X3(1, 150, 2, 5, 8) \
    X3(1, 151, 2, 9, 14) \
    X3(1, 152, 2, 10, 13) \
    X3(1, 153, 2, 10, 15) \
    X3(1, 154, 2, 11, 12) \
    X3(1, 155, 2, 11, 14) \
    X3(1, 156, 3, 3, 9) \
    X3(1, 157, 3, 3, 11) \
    X3(1, 158, 3, 4, 6) \
    X3(1, 159, 3, 5, 7) \
    X3(1, 160, 3, 9, 13) \
    X3(1, 161, 3, 10, 12) \
    X3(1, 162, 3, 11, 13) \
    X3(1, 163, 3, 11, 15) \
    X3(1, 164, 4, 4, 9) \
    X3(1, 165, 4, 4, 11) \
    X3(1, 166, 4, 5, 10) \
    X3(1, 167, 4, 6, 13) \
    X3(1, 168, 4, 6, 15) \
    X3(1, 169, 4, 7, 12) \
    X3(1, 170, 4, 7, 14) \
    X3(1, 171, 4, 8, 15) \
    X3(1, 172, 5, 5, 9) \
    X3(1, 173, 5, 5, 11) \
    X3(1, 174, 5, 6, 12) \
    X3(1, 175, 5, 6, 14) \
    X3(1, 176, 5, 7, 13) \
    X3(1, 177, 5, 7, 15) \
    X3(1, 178, 5, 8, 12) \
    X3(1, 179, 5, 8, 14) \
    X3(1, 180, 6, 6, 11) \
    X3(1, 181, 6, 7, 10) \
    X3(1, 182, 6, 8, 9) \
    X3(1, 183, 6, 8, 11) \
    X3(1, 184, 7, 7, 9) \
    X3(1, 185, 7, 7, 11) \
    X3(1, 186, 7, 8, 10) \
    X3(1, 187, 8, 8, 9) \
    X3(1, 188, 8, 8, 11) \
    X3(1, 189, 9, 9, 11) \
    X3(1, 190, 9, 10, 10) \
    X3(1, 191, 9, 11, 11) \
    X3(1, 192, 9, 12, 14) \
    X3(1, 193, 9, 13, 13) \
    X3(1, 194, 9, 14, 14) \
    X3(1, 195, 10, 10, 11) \
    X3(1, 196, 10, 12, 13) \
    X3(1, 197, 10, 12, 15) \
    X3(1, 198, 10, 14, 15) \
    X3(1, 199, 11, 11, 11) \
    X3(1, 200, 11, 12, 12) \
    X3(1, 201, 11, 12, 14) \
    X3(1, 202, 11, 13, 13) \
    X3(1, 203, 11, 13, 15) \
    X3(1, 204, 11, 14, 14) \
    X3(1, 205, 11, 15, 15) \
    X3(2, 216, 0, 0, 2) \
    X3(2, 217, 0, 1, 5) \
    X3(2, 218, 0, 2, 6) \
    X3(2, 219, 0, 3, 7) \
    X3(2, 220, 0, 4, 10) \
    X3(2, 221, 0, 5, 11) \
    X3(2, 222, 0, 6, 12) \
    X3(2, 223, 0, 7, 13) \
    X3(2, 224, 0, 8, 14) \
    X3(2, 225, 1, 1, 2) \
    X3(2, 226, 1, 1, 12) \
    X3(2, 227, 1, 1, 14) \
    X3(2, 228, 1, 2, 11) \
    X3(2, 229, 1, 3, 10) \
    X3(2, 230, 1, 4, 7) \
    X3(2, 231, 1, 5, 6) \
    X3(2, 232, 1, 5, 8) \
    X3(2, 233, 1, 9, 14) \
    X3(2, 234, 1, 10, 13) \
    X3(2, 235, 1, 10, 15) \
    X3(2, 236, 1, 11, 12) \
    X3(2, 237, 1, 11, 14) \
    X3(2, 238, 2, 2, 2) \
    X3(2, 239, 2, 2, 12) \
    X3(2, 240, 2, 3, 3) \
    X3(2, 241, 2, 3, 13) \
    X3(2, 242, 2, 4, 4) \
    X3(2, 243, 2, 5, 5) \
    X3(2, 244, 2, 6, 6) \
    X3(2, 245, 2, 7, 7) \
    X3(2, 246, 2, 8, 8) \
    X3(2, 247, 2, 9, 9) \
    X3(2, 248, 2, 10, 10) \
    X3(2, 249, 2, 11, 11) \
    X3(2, 250, 2, 12, 12) \
    X3(2, 251, 2, 13, 13) \
    X3(2, 252, 2, 14, 14) \
    X3(2, 253, 2, 15, 15) \
    X3(2, 254, 3, 3, 12) \
    X3(2, 255, 3, 3, 14) \
    X3(2, 256, 3, 4, 5) \
    X3(2, 257, 3, 6, 7) \
    X3(2, 258, 3, 7, 8) \
    X3(2, 259, 3, 9, 10) \
    X3(2, 260, 3, 10, 11) \
    X3(2, 261, 3, 12, 13) \
    X3(2, 262, 3, 13, 14) \
    X3(2, 263, 3, 14, 15) \
    X3(2, 264, 4, 4, 12) \
    X3(2, 265, 4, 5, 13) \
    X3(2, 266, 4, 5, 15) \
    X3(2, 267, 4, 6, 10) \
    X3(2, 268, 4, 7, 9) \
    X3(2, 269, 4, 7, 11) \
    X3(2, 270, 5, 5, 12) \
    X3(2, 271, 5, 5, 14) \
    X3(2, 272, 5, 6, 11) \
    X3(2, 273, 5, 7, 10) \
    X3(2, 274, 5, 8, 9) \
    X3(2, 275, 5, 8, 11) \
    X3(2, 276, 6, 6, 12) \
    X3(2, 277, 6, 7, 13) \
    X3(2, 278, 6, 8, 14) \
    X3(2, 279, 7, 7, 12) \
    X3(2, 280, 7, 7, 14) \
    X3(2, 281, 7, 8, 13) \
    X3(2, 282, 7, 8, 15) \
    X3(2, 283, 8, 8, 12) \
    X3(2, 284, 9, 9, 12) \
    X3(2, 285, 9, 10, 13) \
    X3(2, 286, 9, 11, 14) \
    X3(2, 287, 10, 10, 12) \
    X3(2, 288, 10, 11, 13) \
    X3(2, 289, 10, 11, 15) \
    X3(2, 290, 11, 11, 12) \
    X3(2, 291, 11, 11, 14) \
    X3(2, 292, 12, 12, 12) \
    X3(2, 293, 12, 13, 13) \
    X3(2, 294, 12, 14, 14) \
    X3(2, 295, 12, 15, 15) \
    X3(2, 296, 13, 13, 14) \
    X3(2, 297, 13, 14, 15) \
    X3(3, 312, 0, 0, 3) \
    X3(3, 313, 0, 1, 4) \
    X3(3, 314, 0, 2, 7) \
    X3(3, 315, 0, 3, 6) \
    X3(3, 316, 0, 3, 8) \
    X3(3, 317, 0, 4, 9) \
    X3(3, 318, 0, 4, 11) \
    X3(3, 319, 0, 5, 10) \
    X3(3, 320, 0, 6, 13) \
    X3(3, 321, 0, 7, 12) \
    X3(3, 322, 0, 7, 14) \
    X3(3, 323, 0, 8, 13) \
    X3(3, 324, 0, 8, 15) \
    X3(3, 325, 1, 1, 3) \
    X3(3, 326, 1, 1, 13) \
    X3(3, 327, 1, 1, 15) \
    X3(3, 328, 1, 2, 10) \
    X3(3, 329, 1, 3, 9) \
    X3(3, 330, 1, 3, 11) \
    X3(3, 331, 1, 4, 6) \
    X3(3, 332, 1, 5, 7) \
    X3(3, 333, 1, 9, 13) \
    X3(3, 334, 1, 10, 12) \
    X3(3, 335, 1, 11, 13) \
    X3(3, 336, 1, 11, 15) \
    X3(3, 337, 2, 2, 3) \
    X3(3, 338, 2, 2, 13) \
    X3(3, 339, 2, 3, 12) \
    X3(3, 340, 2, 3, 14) \
    X3(3, 341, 2, 4, 5) \
    X3(3, 342, 2, 6, 7) \
    X3(3, 343, 2, 7, 8) \
    X3(3, 344, 2, 9, 10) \
    X3(3, 345, 2, 10, 11) \
    X3(3, 346, 2, 12, 13) \
    X3(3, 347, 2, 13, 14) \
    X3(3, 348, 2, 14, 15) \
    X3(3, 349, 3, 3, 3) \
    X3(3, 350, 3, 3, 13) \
    X3(3, 351, 3, 3, 15) \
    X3(3, 352, 3, 4, 4) \
    X3(3, 353, 3, 5, 5) \
    X3(3, 354, 3, 6, 6) \
    X3(3, 355, 3, 6, 8) \
    X3(3, 356, 3, 7, 7) \
    X3(3, 357, 3, 8, 8) \
    X3(3, 358, 3, 9, 9) \
    X3(3, 359, 3, 9, 11) \
    X3(3, 360, 3, 10, 10) \
    X3(3, 361, 3, 11, 11) \
    X3(3, 362, 3, 12, 12) \
    X3(3, 363, 3, 12, 14) \
    X3(3, 364, 3, 13, 13) \
    X3(3, 365, 3, 13, 15) \
    X3(3, 366, 3, 14, 14) \
    X3(3, 367, 3, 15, 15) \
    X3(3, 368, 4, 4, 13) \
    X3(3, 369, 4, 4, 15) \
    X3(3, 370, 4, 5, 12) \
    X3(3, 371, 4, 5, 14) \
    X3(3, 372, 4, 6, 9) \
    X3(3, 373, 4, 6, 11) \
    X3(3, 374, 4, 7, 10) \
    X3(3, 375, 4, 8, 9) \
    X3(3, 376, 5, 5, 13) \
    X3(3, 377, 5, 5, 15) \
    X3(3, 378, 5, 6, 10) \
    X3(3, 379, 5, 7, 9) \
    X3(3, 380, 5, 7, 11) \
    X3(3, 381, 5, 8, 10) \
    X3(3, 382, 6, 6, 13) \
    X3(3, 383, 6, 7, 12) \
    X3(3, 384, 6, 7, 14) \
    X3(3, 385, 6, 8, 13) \
    X3(3, 386, 6, 8, 15) \
    X3(3, 387, 7, 7, 13) \
    X3(3, 388, 7, 7, 15) \
    X3(3, 389, 7, 8, 12) \
    X3(3, 390, 7, 8, 14) \
    X3(3, 391, 8, 8, 13) \
    X3(3, 392, 8, 8, 15) \
    X3(3, 393, 9, 9, 13) \
    X3(3, 394, 9, 10, 12) \
    X3(3, 395, 9, 10, 14) \
    X3(3, 396, 9, 11, 13) \
    X3(3, 397, 10, 10, 13) \
    X3(3, 398, 10, 10, 15) \
    X3(3, 399, 10, 11, 12) \
    X3(3, 400, 11, 11, 13) \
    X3(3, 401, 11, 11, 15) \
    X3(3, 402, 12, 12, 13) \
    X3(3, 403, 12, 13, 14) \
    X3(3, 404, 12, 14, 15) \
    X3(3, 405, 13, 13, 13) \
    X3(3, 406, 13, 13, 15) \
    X3(3, 407, 13, 14, 14) \
    X3(3, 408, 13, 15, 15) \
    X3(3, 409, 14, 14, 15) \
    X3(4, 424, 0, 0, 4) \
    X3(4, 425, 0, 1, 3) \
    X3(4, 426, 0, 1, 13) \
    X3(4, 427, 0, 1, 15) \
    X3(4, 428, 0, 2, 10) \
    X3(4, 429, 0, 3, 9) \
    X3(4, 430, 0, 3, 11) \
    X3(4, 431, 0, 4, 6) \
    X3(4, 432, 0, 5, 7) \
    X3(4, 433, 0, 9, 13) \
    X3(4, 434, 0, 10, 12) \
    X3(4, 435, 0, 11, 13) \
    X3(4, 436, 0, 11, 15) \
    X3(4, 437, 1, 1, 4) \
    X3(4, 438, 1, 2, 7) \
    X3(4, 439, 1, 3, 6) \
    X3(4, 440, 1, 4, 9) \
    X3(4, 441, 1, 4, 11) \
    X3(4, 442, 1, 5, 10) \
    X3(4, 443, 1, 6, 13) \
    X3(4, 444, 1, 6, 15) \
    X3(4, 445, 1, 7, 12) \
    X3(4, 446, 1, 7, 14) \
    X3(4, 447, 1, 8, 13) \
    X3(4, 448, 1, 8, 15) \
    X3(4, 449, 2, 2, 4) \
    X3(4, 450, 2, 3, 5) \
    X3(4, 451, 2, 4, 12) \
    X3(4, 452, 2, 5, 13) \
    X3(4, 453, 2, 5, 15) \
    X3(4, 454, 2, 6, 10) \
    X3(4, 455, 2, 7, 9) \
    X3(4, 456, 2, 7, 11) \
    X3(4, 457, 3, 3, 4) \
    X3(4, 458, 3, 4, 13) \
    X3(4, 459, 3, 4, 15) \
    X3(4, 460, 3, 5, 12) \
    X3(4, 461, 3, 5, 14) \
    X3(4, 462, 3, 6, 9) \
    X3(4, 463, 3, 6, 11) \
    X3(4, 464, 3, 7, 10) \
    X3(4, 465, 3, 8, 9) \
    X3(4, 466, 3, 8, 11) \
    X3(4, 467, 4, 4, 4) \
    X3(4, 468, 4, 5, 5) \
    X3(4, 469, 4, 6, 6) \
    X3(4, 470, 4, 7, 7) \
    X3(4, 471, 4, 8, 8) \
    X3(4, 472, 4, 9, 9) \
    X3(4, 473, 4, 9, 11) \
    X3(4, 474, 4, 10, 10) \
    X3(4, 475, 4, 11, 11) \
    X3(4, 476, 4, 12, 12) \
    X3(4, 477, 4, 13, 13) \
    X3(4, 478, 4, 13, 15) \
    X3(4, 479, 4, 14, 14) \
    X3(4, 480, 4, 15, 15) \
    X3(4, 481, 5, 9, 10) \
    X3(4, 482, 5, 10, 11) \
    X3(4, 483, 5, 12, 13) \
    X3(4, 484, 5, 12, 15) \
    X3(4, 485, 5, 13, 14) \
    X3(4, 486, 5, 14, 15) \
    X3(4, 487, 6, 9, 13) \
    X3(4, 488, 6, 10, 12) \
    X3(4, 489, 6, 11, 13) \
    X3(4, 490, 6, 11, 15) \
    X3(4, 491, 7, 9, 12) \
    X3(4, 492, 7, 9, 14) \
    X3(4, 493, 7, 10, 13) \
    X3(4, 494, 7, 10, 15) \
    X3(4, 495, 7, 11, 12) \
    X3(4, 496, 7, 11, 14) \
    X3(4, 497, 8, 9, 13) \
    X3(4, 498, 8, 10, 14) \
    X3(4, 499, 8, 11, 15) \
    X3(5, 515, 0, 0, 5) \
    X3(5, 516, 0, 1, 2) \
    X3(5, 517, 0, 1, 12) \
    X3(5, 518, 0, 1, 14) \
    X3(5, 519, 0, 2, 11) \
    X3(5, 520, 0, 3, 10) \
    X3(5, 521, 0, 4, 7) \
    X3(5, 522, 0, 5, 6) \
    X3(5, 523, 0, 5, 8) \
    X3(5, 524, 0, 9, 14) \
    X3(5, 525, 0, 10, 13) \
    X3(5, 526, 0, 10, 15) \
    X3(5, 527, 0, 11, 12) \
    X3(5, 528, 0, 11, 14) \
    X3(5, 529, 1, 1, 5) \
    X3(5, 530, 1, 2, 6) \
    X3(5, 531, 1, 2, 8) \
    X3(5, 532, 1, 3, 7) \
    X3(5, 533, 1, 4, 10) \
    X3(5, 534, 1, 5, 9) \
    X3(5, 535, 1, 5, 11) \
    X3(5, 536, 1, 6, 12) \
    X3(5, 537, 1, 6, 14) \
    X3(5, 538, 1, 7, 13) \
    X3(5, 539, 1, 7, 15) \
    X3(5, 540, 1, 8, 12) \
    X3(5, 541, 1, 8, 14) \
    X3(5, 542, 2, 2, 5) \
    X3(5, 543, 2, 3, 4) \
    X3(5, 544, 2, 4, 13) \
    X3(5, 545, 2, 4, 15) \
    X3(5, 546, 2, 5, 12) \
    X3(5, 547, 2, 5, 14) \
    X3(5, 548, 2, 6, 11) \
    X3(5, 549, 2, 7, 10) \
    X3(5, 550, 2, 8, 9) \
    X3(5, 551, 2, 8, 11) \
    X3(5, 552, 3, 3, 5) \
    X3(5, 553, 3, 4, 12) \
    X3(5, 554, 3, 4, 14) \
    X3(5, 555, 3, 5, 13) \
    X3(5, 556, 3, 5, 15) \
    X3(5, 557, 3, 6, 10) \
    X3(5, 558, 3, 7, 9) \
    X3(5, 559, 3, 7, 11) \
    X3(5, 560, 3, 8, 10) \
    X3(5, 561, 4, 4, 5) \
    X3(5, 562, 4, 9, 10) \
    X3(5, 563, 4, 10, 11) \
    X3(5, 564, 4, 12, 13) \
    X3(5, 565, 4, 12, 15) \
    X3(5, 566, 4, 13, 14) \
    X3(5, 567, 4, 14, 15) \
    X3(5, 568, 5, 5, 5) \
    X3(5, 569, 5, 6, 6) \
    X3(5, 570, 5, 7, 7) \
    X3(5, 571, 5, 8, 8) \
    X3(5, 572, 5, 9, 9) \
    X3(5, 573, 5, 9, 11) \
    X3(5, 574, 5, 10, 10) \
    X3(5, 575, 5, 11, 11) \
    X3(5, 576, 5, 12, 12) \
    X3(5, 577, 5, 12, 14) \
    X3(5, 578, 5, 13, 13) \
    X3(5, 579, 5, 13, 15) \
    X3(5, 580, 5, 14, 14) \
    X3(5, 581, 5, 15, 15) \
    X3(5, 582, 6, 9, 14) \
    X3(5, 583, 6, 10, 13) \
    X3(5, 584, 6, 10, 15) \
    X3(5, 585, 6, 11, 12) \
    X3(5, 586, 6, 11, 14) \
    X3(5, 587, 7, 9, 13) \
    X3(5, 588, 7, 10, 12) \
    X3(5, 589, 7, 11, 13) \
    X3(5, 590, 7, 11, 15) \
    X3(5, 591, 8, 9, 12) \
    X3(5, 592, 8, 9, 14) \
    X3(5, 593, 8, 10, 13) \
    X3(5, 594, 8, 10, 15) \
    X3(5, 595, 8, 11, 12) \
    X3(5, 596, 8, 11, 14) \
    X3(6, 615, 0, 0, 6) \
    X3(6, 616, 0, 1, 1) \
    X3(6, 617, 0, 1, 11) \
    X3(6, 618, 0, 2, 2) \
    X3(6, 619, 0, 2, 12) \
    X3(6, 620, 0, 3, 3) \
    X3(6, 621, 0, 3, 13) \
    X3(6, 622, 0, 4, 4) \
    X3(6, 623, 0, 5, 5) \
    X3(6, 624, 0, 6, 6) \
    X3(6, 625, 0, 7, 7) \
    X3(6, 626, 0, 8, 8) \
    X3(6, 627, 0, 9, 9) \
    X3(6, 628, 0, 11, 11) \
    X3(6, 629, 0, 12, 12) \
    X3(6, 630, 0, 13, 13) \
    X3(6, 631, 0, 15, 15) \
    X3(6, 632, 1, 1, 6) \
    X3(6, 633, 1, 1, 8) \
    X3(6, 634, 1, 2, 5) \
    X3(6, 635, 1, 3, 4) \
    X3(6, 636, 1, 4, 13) \
    X3(6, 637, 1, 4, 15) \
    X3(6, 638, 1, 5, 12) \
    X3(6, 639, 1, 5, 14) \
    X3(6, 640, 1, 6, 11) \
    X3(6, 641, 1, 7, 10) \
    X3(6, 642, 1, 8, 9) \
    X3(6, 643, 1, 8, 11) \
    X3(6, 644, 2, 2, 6) \
    X3(6, 645, 2, 3, 7) \
    X3(6, 646, 2, 4, 10) \
    X3(6, 647, 2, 5, 11) \
    X3(6, 648, 2, 6, 12) \
    X3(6, 649, 2, 7, 13) \
    X3(6, 650, 2, 8, 14) \
    X3(6, 651, 3, 3, 6) \
    X3(6, 652, 3, 3, 8) \
    X3(6, 653, 3, 4, 9) \
    X3(6, 654, 3, 4, 11) \
    X3(6, 655, 3, 5, 10) \
    X3(6, 656, 3, 6, 13) \
    X3(6, 657, 3, 7, 12) \
    X3(6, 658, 3, 7, 14) \
    X3(6, 659, 3, 8, 13) \
    X3(6, 660, 3, 8, 15) \
    X3(6, 661, 4, 4, 6) \
    X3(6, 662, 4, 9, 13) \
    X3(6, 663, 4, 10, 12) \
    X3(6, 664, 4, 11, 13) \
    X3(6, 665, 4, 11, 15) \
    X3(6, 666, 5, 5, 6) \
    X3(6, 667, 5, 9, 14) \
    X3(6, 668, 5, 10, 13) \
    X3(6, 669, 5, 10, 15) \
    X3(6, 670, 5, 11, 12) \
    X3(6, 671, 5, 11, 14) \
    X3(6, 672, 6, 6, 6) \
    X3(6, 673, 6, 7, 7) \
    X3(6, 674, 6, 8, 8) \
    X3(6, 675, 6, 9, 9) \
    X3(6, 676, 6, 10, 10) \
    X3(6, 677, 6, 11, 11) \
    X3(6, 678, 6, 12, 12) \
    X3(6, 679, 6, 13, 13) \
    X3(6, 680, 6, 14, 14) \
    X3(6, 681, 6, 15, 15) \
    X3(6, 682, 7, 9, 10) \
    X3(6, 683, 7, 10, 11) \
    X3(6, 684, 7, 12, 13) \
    X3(6, 685, 7, 13, 14) \
    X3(6, 686, 7, 14, 15) \
    X3(6, 687, 8, 9, 11) \
    X3(6, 688, 8, 11, 11) \
    X3(6, 689, 8, 12, 14) \
    X3(6, 690, 8, 13, 13) \
    X3(6, 691, 8, 13, 15) \
    X3(7, 707, 0, 0, 7) \
    X3(7, 708, 0, 1, 10) \
    X3(7, 709, 0, 2, 3) \
    X3(7, 710, 0, 2, 13) \
    X3(7, 711, 0, 3, 12) \
    X3(7, 712, 0, 3, 14) \
    X3(7, 713, 0, 4, 5) \
    X3(7, 714, 0, 6, 7) \
    X3(7, 715, 0, 7, 8) \
    X3(7, 716, 0, 9, 10) \
    X3(7, 717, 0, 10, 11) \
    X3(7, 718, 0, 12, 13) \
    X3(7, 719, 0, 13, 14) \
    X3(7, 720, 0, 14, 15) \
    X3(7, 721, 1, 1, 7) \
    X3(7, 722, 1, 2, 4) \
    X3(7, 723, 1, 3, 5) \
    X3(7, 724, 1, 4, 12) \
    X3(7, 725, 1, 4, 14) \
    X3(7, 726, 1, 5, 13) \
    X3(7, 727, 1, 5, 15) \
    X3(7, 728, 1, 6, 10) \
    X3(7, 729, 1, 7, 9) \
    X3(7, 730, 1, 7, 11) \
    X3(7, 731, 1, 8, 10) \
    X3(7, 732, 2, 2, 7) \
    X3(7, 733, 2, 3, 6) \
    X3(7, 734, 2, 3, 8) \
    X3(7, 735, 2, 4, 9) \
    X3(7, 736, 2, 4, 11) \
    X3(7, 737, 2, 5, 10) \
    X3(7, 738, 2, 6, 13) \
    X3(7, 739, 2, 7, 12) \
    X3(7, 740, 2, 7, 14) \
    X3(7, 741, 2, 8, 13) \
    X3(7, 742, 2, 8, 15) \
    X3(7, 743, 3, 3, 7) \
    X3(7, 744, 3, 4, 10) \
    X3(7, 745, 3, 5, 9) \
    X3(7, 746, 3, 5, 11) \
    X3(7, 747, 3, 6, 12) \
    X3(7, 748, 3, 6, 14) \
    X3(7, 749, 3, 7, 13) \
    X3(7, 750, 3, 7, 15) \
    X3(7, 751, 3, 8, 12) \
    X3(7, 752, 3, 8, 14) \
    X3(7, 753, 4, 4, 7) \
    X3(7, 754, 4, 9, 12) \
    X3(7, 755, 4, 9, 14) \
    X3(7, 756, 4, 10, 13) \
    X3(7, 757, 4, 10, 15) \
    X3(7, 758, 4, 11, 12) \
    X3(7, 759, 4, 11, 14) \
    X3(7, 760, 5, 5, 7) \
    X3(7, 761, 5, 9, 13) \
    X3(7, 762, 5, 10, 12) \
    X3(7, 763, 5, 11, 13) \
    X3(7, 764, 5, 11, 15) \
    X3(7, 765, 6, 6, 7) \
    X3(7, 766, 6, 9, 10) \
    X3(7, 767, 6, 10, 11) \
    X3(7, 768, 6, 12, 13) \
    X3(7, 769, 6, 13, 14) \
    X3(7, 770, 6, 14, 15) \
    X3(7, 771, 7, 7, 7) \
    X3(7, 772, 7, 8, 8) \
    X3(7, 773, 7, 9, 9) \
    X3(7, 774, 7, 9, 11) \
    X3(7, 775, 7, 10, 10) \
    X3(7, 776, 7, 11, 11) \
    X3(7, 777, 7, 12, 12) \
    X3(7, 778, 7, 12, 14) \
    X3(7, 779, 7, 13, 13) \
    X3(7, 780, 7, 13, 15) \
    X3(7, 781, 7, 14, 14) \
    X3(7, 782, 7, 15, 15) \
    X3(7, 783, 8, 9, 10) \
    X3(7, 784, 8, 10, 11) \
    X3(7, 785, 8, 12, 13) \
    X3(7, 786, 8, 12, 15) \
    X3(7, 787, 8, 13, 14) \
    X3(7, 788, 8, 14, 15) \
    X3(8, 806, 0, 0, 8) \
    X3(8, 807, 0, 1, 1) \
    X3(8, 808, 0, 1, 9) \
    X3(8, 809, 0, 1, 11) \
    X3(8, 810, 0, 2, 14) \
    X3(8, 811, 0, 3, 3) \
    X3(8, 812, 0, 3, 13) \
    X3(8, 813, 0, 3, 15) \
    X3(8, 814, 0, 5, 5) \
    X3(8, 815, 0, 6, 8) \
    X3(8, 816, 0, 7, 7) \
    X3(8, 817, 0, 9, 11) \
    X3(8, 818, 0, 11, 11) \
    X3(8, 819, 0, 12, 14) \
    X3(8, 820, 0, 13, 13) \
    X3(8, 821, 0, 13, 15) \
    X3(8, 822, 1, 1, 6) \
    X3(8, 823, 1, 1, 8) \
    X3(8, 824, 1, 2, 5) \
    X3(8, 825, 1, 4, 13) \
    X3(8, 826, 1, 4, 15) \
    X3(8, 827, 1, 5, 12) \
    X3(8, 828, 1, 5, 14) \
    X3(8, 829, 1, 6, 9) \
    X3(8, 830, 1, 6, 11) \
    X3(8, 831, 1, 7, 10) \
    X3(8, 832, 1, 8, 9) \
    X3(8, 833, 1, 8, 11) \
    X3(8, 834, 2, 2, 8) \
    X3(8, 835, 2, 3, 7) \
    X3(8, 836, 2, 5, 9) \
    X3(8, 837, 2, 5, 11) \
    X3(8, 838, 2, 6, 14) \
    X3(8, 839, 2, 7, 13) \
    X3(8, 840, 2, 7, 15) \
    X3(8, 841, 2, 8, 12) \
    X3(8, 842, 3, 3, 6) \
    X3(8, 843, 3, 3, 8) \
    X3(8, 844, 3, 4, 9) \
    X3(8, 845, 3, 4, 11) \
    X3(8, 846, 3, 5, 10) \
    X3(8, 847, 3, 6, 13) \
    X3(8, 848, 3, 6, 15) \
    X3(8, 849, 3, 7, 12) \
    X3(8, 850, 3, 7, 14) \
    X3(8, 851, 3, 8, 13) \
    X3(8, 852, 3, 8, 15) \
    X3(8, 853, 4, 4, 8) \
    X3(8, 854, 4, 9, 13) \
    X3(8, 855, 4, 10, 14) \
    X3(8, 856, 4, 11, 15) \
    X3(8, 857, 5, 5, 8) \
    X3(8, 858, 5, 9, 12) \
    X3(8, 859, 5, 9, 14) \
    X3(8, 860, 5, 10, 13) \
    X3(8, 861, 5, 10, 15) \
    X3(8, 862, 5, 11, 12) \
    X3(8, 863, 5, 11, 14) \
    X3(8, 864, 6, 6, 8) \
    X3(8, 865, 6, 9, 11) \
    X3(8, 866, 6, 11, 11) \
    X3(8, 867, 6, 12, 14) \
    X3(8, 868, 6, 13, 13) \
    X3(8, 869, 6, 13, 15) \
    X3(8, 870, 7, 7, 8) \
    X3(8, 871, 7, 9, 10) \
    X3(8, 872, 7, 10, 11) \
    X3(8, 873, 7, 12, 13) \
    X3(8, 874, 7, 12, 15) \
    X3(8, 875, 7, 13, 14) \
    X3(8, 876, 7, 14, 15) \
    X3(8, 877, 8, 8, 8) \
    X3(8, 878, 8, 9, 9) \
    X3(8, 879, 8, 9, 11) \
    X3(8, 880, 8, 10, 10) \
    X3(8, 881, 8, 11, 11) \
    X3(8, 882, 8, 12, 12) \
    X3(8, 883, 8, 13, 13) \
    X3(8, 884, 8, 13, 15) \
    X3(8, 885, 8, 14, 14) \
    X3(8, 886, 8, 15, 15)
#define SXB_S2_M1_NUM_TERMS 94
#define SXB_S2_M1_TERMS(X1, X2, X3) \
    X1(0, 0, 0) \
    X2(0, 1, 0, 0) \
    X2(0, 2, 1, 1) \
    X2(0, 3, 2, 2) \
    X2(0, 4, 3, 3) \
    X2(0, 5, 4, 4) \
    X2(0, 6, 5, 5) \
    X2(0, 7, 6, 6) \
    X2(0, 8, 7, 7) \
    X2(0, 9, 8, 8) \
    X2(0, 10, 9, 9) \
    X2(0, 11, 10, 10) \
    X2(0, 12, 11, 11) \
    X2(0, 13, 12, 12) \
    X2(0, 14, 13, 13) \
    X2(0, 15, 14, 14) \
    X2(0, 16, 15, 15) \
    X3(0, 17, 0, 0, 0) \
    X3(0, 18, 0, 1, 1) \
    X3(0, 19, 0, 2, 2) \
    X3(0, 20, 0, 3, 3) \
    X3(0, 21, 0, 4, 4) \
    X3(0, 22, 0, 5, 5) \
    X3(0, 23, 0, 6, 6) \
    X3(0, 24, 0, 7, 7) \
    X3(0, 25, 0, 8, 8) \
    X3(0, 26, 0, 9, 9) \
    X3(0, 27, 0, 10, 10) \
    X3(0, 28, 0, 11, 11) \
    X3(0, 29, 0, 12, 12) \
    X3(0, 30, 0, 13, 13) \
    X3(0, 31, 0, 14, 14) \
    X3(0, 32, 0, 15, 15) \
    X3(0, 33, 1, 1, 6) \
    X3(0, 34, 1, 1, 8) \
    X3(0, 35, 1, 2, 5) \
    X3(0, 36, 1, 3, 4) \
    X3(0, 37, 1, 4, 13) \
    X3(0, 38, 1, 4, 15) \
    X3(0, 39, 1, 5, 12) \
    X3(0, 40, 1, 5, 14) \
    X3(0, 41, 1, 6, 11) \
    X3(0, 42, 1, 7, 10) \
    X3(0, 43, 1, 8, 9) \
    X3(0, 44, 1, 8, 11) \
    X3(0, 45, 2, 2, 6) \
    X3(0, 46, 2, 3, 7) \
    X3(0, 47, 2, 4, 10) \
    X3(0, 48, 2, 5, 11) \
    X3(0, 49, 2, 6, 12) \
    X3(0, 50, 2, 7, 13) \
    X3(0, 51, 2, 8, 14) \
    X3(0, 52, 3, 3, 6) \
    X3(0, 53, 3, 3, 8) \
    X3(0, 54, 3, 4, 9) \
    X3(0, 55, 3, 4, 11) \
    X3(0, 56, 3, 5, 10) \
    X3(0, 57, 3, 6, 13) \
    X3(0, 58, 3, 7, 12) \
    X3(0, 59, 3, 7, 14) \
    X3(0, 60, 3, 8, 13) \
    X3(0, 61, 3, 8, 15) \
    X3(0, 62, 4, 4, 6) \
    X3(0, 63, 4, 5, 7) \
    X3(0, 64, 4, 9, 13) \
    X3(0, 65, 4, 10, 12) \
    X3(0, 66, 4, 11, 13) \
    X3(0, 67, 4, 11, 15) \
    X3(0, 68, 5, 5, 6) \
    X3(0, 69, 5, 5, 8) \
    X3(0, 70, 5, 9, 14) \
    X3(0, 71, 5, 10, 13) \
    X3(0, 72, 5, 10, 15) \
    X3(0, 73, 5, 11, 12) \
    X3(0, 74, 5, 11, 14) \
    X3(0, 75, 6, 6, 6) \
    X3(0, 76, 6, 7, 7) \
    X3(0, 77, 6, 8, 8) \
    X3(0, 78, 6, 9, 9) \
    X3(0, 79, 6, 11, 11) \
    X3(0, 80, 6, 12, 12) \
    X3(0, 81, 6, 13, 13) \
    X3(0, 82, 6, 15, 15) \
    X3(0, 83, 7, 7, 8) \
    X3(0, 84, 7, 9, 10) \
    X3(0, 85, 7, 10, 11) \
    X3(0, 86, 7, 12, 13) \
    X3(0, 87, 7, 13, 14) \
    X3(0, 88, 7, 14, 15) \
    X3(0, 89, 8, 9, 11) \
    X3(0, 90, 8, 11, 11) \
    X3(0, 91, 8, 12, 14) \
    X3(0, 92, 8, 13, 13) \
    X3(0, 93, 8, 13, 15)
#define SXB_S2_M0_FORWARD_BODY \
      o[0] = f2_fma(W(0), x[0], o[0]); \
      o[1] = f2_fma(W(94), x[1], o[1]); \
      o[2] = f2_fma(W(206), x[2], o[2]); \
      o[3] = f2_fma(W(298), x[3], o[3]); \
      o[4] = f2_fma(W(410), x[4], o[4]); \
      o[5] = f2_fma(W(500), x[5], o[5]); \
      o[6] = f2_fma(W(597), x[6], o[6]); \
      o[7] = f2_fma(W(692), x[7], o[7]); \
      o[8] = f2_fma(W(789), x[8], o[8]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); o[0] = f2_fma(p, f2_fma(W(17), x[0], W(1)), o[0]); o[1] = f2_fma(p, f2_mul(W(108), x[1]), o[1]); o[2] = f2_fma(p, f2_mul(W(216), x[2]), o[2]); o[3] = f2_fma(p, f2_mul(W(312), x[3]), o[3]); o[4] = f2_fma(p, f2_mul(W(424), x[4]), o[4]); o[5] = f2_fma(p, f2_mul(W(515), x[5]), o[5]); o[6] = f2_fma(p, f2_mul(W(615), x[6]), o[6]); o[7] = f2_fma(p, f2_mul(W(707), x[7]), o[7]); o[8] = f2_fma(p, f2_mul(W(806), x[8]), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); o[0] = f2_fma(p, f2_mul(W(18), x[1]), o[0]); o[1] = f2_fma(p, f2_fma(W(110), x[8], f2_fma(W(109), x[6], W(95))), o[1]); o[2] = f2_fma(p, f2_mul(W(217), x[5]), o[2]); o[3] = f2_fma(p, f2_mul(W(313), x[4]), o[3]); o[4] = f2_fma(p, f2_fma(W(427), x[15], f2_fma(W(426), x[13], f2_mul(W(425), x[3]))), o[4]); o[5] = f2_fma(p, f2_fma(W(518), x[14], f2_fma(W(517), x[12], f2_mul(W(516), x[2]))), o[5]); o[6] = f2_fma(p, f2_fma(W(617), x[11], f2_mul(W(616), x[1])), o[6]); o[7] = f2_fma(p, f2_mul(W(708), x[10]), o[7]); o[8] = f2_fma(p, f2_fma(W(809), x[11], f2_fma(W(808), x[9], f2_mul(W(807), x[1]))), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); o[0] = f2_fma(p, f2_mul(W(19), x[2]), o[0]); o[1] = f2_fma(p, f2_mul(W(111), x[5]), o[1]); o[2] = f2_fma(p, f2_fma(W(218), x[6], W(207)), o[2]); o[3] = f2_fma(p, f2_mul(W(314), x[7]), o[3]); o[4] = f2_fma(p, f2_mul(W(428), x[10]), o[4]); o[5] = f2_fma(p, f2_mul(W(519), x[11]), o[5]); o[6] = f2_fma(p, f2_fma(W(619), x[12], f2_mul(W(618), x[2])), o[6]); o[7] = f2_fma(p, f2_fma(W(710), x[13], f2_mul(W(709), x[3])), o[7]); o[8] = f2_fma(p, f2_mul(W(810), x[14]), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); o[0] = f2_fma(p, f2_mul(W(20), x[3]), o[0]); o[1] = f2_fma(p, f2_mul(W(112), x[4]), o[1]); o[2] = f2_fma(p, f2_mul(W(219), x[7]), o[2]); o[3] = f2_fma(p, f2_fma(W(316), x[8], f2_fma(W(315), x[6], W(299))), o[3]); o[4] = f2_fma(p, f2_fma(W(430), x[11], f2_mul(W(429), x[9])), o[4]); o[5] = f2_fma(p, f2_mul(W(520), x[10]), o[5]); o[6] = f2_fma(p, f2_fma(W(621), x[13], f2_mul(W(620), x[3])), o[6]); o[7] = f2_fma(p, f2_fma(W(712), x[14], f2_mul(W(711), x[12])), o[7]); o[8] = f2_fma(p, f2_fma(W(813), x[15], f2_fma(W(812), x[13], f2_mul(W(811), x[3]))), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); o[0] = f2_fma(p, f2_mul(W(21), x[4]), o[0]); o[1] = f2_fma(p, f2_fma(W(114), x[15], f2_mul(W(113), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(220), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(318), x[11], f2_mul(W(317), x[9])), o[3]); o[4] = f2_fma(p, f2_fma(W(431), x[6], W(411)), o[4]); o[5] = f2_fma(p, f2_mul(W(521), x[7]), o[5]); o[6] = f2_fma(p, f2_mul(W(622), x[4]), o[6]); o[7] = f2_fma(p, f2_mul(W(713), x[5]), o[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); o[0] = f2_fma(p, f2_mul(W(22), x[5]), o[0]); o[1] = f2_fma(p, f2_fma(W(116), x[14], f2_mul(W(115), x[12])), o[1]); o[2] = f2_fma(p, f2_mul(W(221), x[11]), o[2]); o[3] = f2_fma(p, f2_mul(W(319), x[10]), o[3]); o[4] = f2_fma(p, f2_mul(W(432), x[7]), o[4]); o[5] = f2_fma(p, f2_fma(W(523), x[8], f2_fma(W(522), x[6], W(501))), o[5]); o[6] = f2_fma(p, f2_mul(W(623), x[5]), o[6]); o[8] = f2_fma(p, f2_mul(W(814), x[5]), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); o[0] = f2_fma(p, f2_mul(W(23), x[6]), o[0]); o[1] = f2_fma(p, f2_mul(W(117), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(222), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(320), x[13]), o[3]); o[6] = f2_fma(p, f2_fma(W(624), x[6], W(598)), o[6]); o[7] = f2_fma(p, f2_mul(W(714), x[7]), o[7]); o[8] = f2_fma(p, f2_mul(W(815), x[8]), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); o[0] = f2_fma(p, f2_mul(W(24), x[7]), o[0]); o[1] = f2_fma(p, f2_mul(W(118), x[10]), o[1]); o[2] = f2_fma(p, f2_mul(W(223), x[13]), o[2]); o[3] = f2_fma(p, f2_fma(W(322), x[14], f2_mul(W(321), x[12])), o[3]); o[6] = f2_fma(p, f2_mul(W(625), x[7]), o[6]); o[7] = f2_fma(p, f2_fma(W(715), x[8], W(693)), o[7]); o[8] = f2_fma(p, f2_mul(W(816), x[7]), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); o[0] = f2_fma(p, f2_mul(W(25), x[8]), o[0]); o[1] = f2_fma(p, f2_fma(W(120), x[11], f2_mul(W(119), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(224), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(324), x[15], f2_mul(W(323), x[13])), o[3]); o[6] = f2_fma(p, f2_mul(W(626), x[8]), o[6]); o[8] = f2_fma(p, W(790), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); o[0] = f2_fma(p, f2_mul(W(26), x[9]), o[0]); o[4] = f2_fma(p, f2_mul(W(433), x[13]), o[4]); o[5] = f2_fma(p, f2_mul(W(524), x[14]), o[5]); o[6] = f2_fma(p, f2_mul(W(627), x[9]), o[6]); o[7] = f2_fma(p, f2_mul(W(716), x[10]), o[7]); o[8] = f2_fma(p, f2_mul(W(817), x[11]), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); o[0] = f2_fma(p, f2_mul(W(27), x[10]), o[0]); o[4] = f2_fma(p, f2_mul(W(434), x[12]), o[4]); o[5] = f2_fma(p, f2_fma(W(526), x[15], f2_mul(W(525), x[13])), o[5]); o[7] = f2_fma(p, f2_mul(W(717), x[11]), o[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); o[0] = f2_fma(p, f2_mul(W(28), x[11]), o[0]); o[4] = f2_fma(p, f2_fma(W(436), x[15], f2_mul(W(435), x[13])), o[4]); o[5] = f2_fma(p, f2_fma(W(528), x[14], f2_mul(W(527), x[12])), o[5]); o[6] = f2_fma(p, f2_mul(W(628), x[11]), o[6]); o[8] = f2_fma(p, f2_mul(W(818), x[11]), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); o[0] = f2_fma(p, f2_mul(W(29), x[12]), o[0]); o[6] = f2_fma(p, f2_mul(W(629), x[12]), o[6]); o[7] = f2_fma(p, f2_mul(W(718), x[13]), o[7]); o[8] = f2_fma(p, f2_mul(W(819), x[14]), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); o[0] = f2_fma(p, f2_mul(W(30), x[13]), o[0]); o[6] = f2_fma(p, f2_mul(W(630), x[13]), o[6]); o[7] = f2_fma(p, f2_mul(W(719), x[14]), o[7]); o[8] = f2_fma(p, f2_fma(W(821), x[15], f2_mul(W(820), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); o[0] = f2_fma(p, f2_mul(W(31), x[14]), o[0]); o[7] = f2_fma(p, f2_mul(W(720), x[15]), o[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); o[0] = f2_fma(p, f2_mul(W(32), x[15]), o[0]); o[6] = f2_fma(p, f2_mul(W(631), x[15]), o[6]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); o[0] = f2_fma(p, f2_fma(W(34), x[8], f2_fma(W(33), x[6], W(2))), o[0]); o[1] = f2_fma(p, f2_fma(W(123), x[11], f2_fma(W(122), x[9], f2_mul(W(121), x[1]))), o[1]); o[2] = f2_fma(p, f2_fma(W(227), x[14], f2_fma(W(226), x[12], f2_mul(W(225), x[2]))), o[2]); o[3] = f2_fma(p, f2_fma(W(327), x[15], f2_fma(W(326), x[13], f2_mul(W(325), x[3]))), o[3]); o[4] = f2_fma(p, f2_mul(W(437), x[4]), o[4]); o[5] = f2_fma(p, f2_mul(W(529), x[5]), o[5]); o[6] = f2_fma(p, f2_fma(W(633), x[8], f2_fma(W(632), x[6], W(599))), o[6]); o[7] = f2_fma(p, f2_mul(W(721), x[7]), o[7]); o[8] = f2_fma(p, f2_fma(W(823), x[8], f2_fma(W(822), x[6], W(791))), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); o[0] = f2_fma(p, f2_mul(W(35), x[5]), o[0]); o[1] = f2_fma(p, f2_fma(W(126), x[14], f2_fma(W(125), x[12], f2_mul(W(124), x[2]))), o[1]); o[2] = f2_fma(p, f2_mul(W(228), x[11]), o[2]); o[3] = f2_fma(p, f2_mul(W(328), x[10]), o[3]); o[4] = f2_fma(p, f2_mul(W(438), x[7]), o[4]); o[5] = f2_fma(p, f2_fma(W(531), x[8], f2_fma(W(530), x[6], W(502))), o[5]); o[6] = f2_fma(p, f2_mul(W(634), x[5]), o[6]); o[7] = f2_fma(p, f2_mul(W(722), x[4]), o[7]); o[8] = f2_fma(p, f2_mul(W(824), x[5]), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); o[0] = f2_fma(p, f2_mul(W(36), x[4]), o[0]); o[1] = f2_fma(p, f2_fma(W(129), x[15], f2_fma(W(128), x[13], f2_mul(W(127), x[3]))), o[1]); o[2] = f2_fma(p, f2_mul(W(229), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(330), x[11], f2_mul(W(329), x[9])), o[3]); o[4] = f2_fma(p, f2_fma(W(439), x[6], W(412)), o[4]); o[5] = f2_fma(p, f2_mul(W(532), x[7]), o[5]); o[6] = f2_fma(p, f2_mul(W(635), x[4]), o[6]); o[7] = f2_fma(p, f2_mul(W(723), x[5]), o[7]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); o[0] = f2_fma(p, f2_fma(W(38), x[15], f2_mul(W(37), x[13])), o[0]); o[1] = f2_fma(p, f2_mul(W(130), x[4]), o[1]); o[2] = f2_fma(p, f2_mul(W(230), x[7]), o[2]); o[3] = f2_fma(p, f2_fma(W(331), x[6], W(300)), o[3]); o[4] = f2_fma(p, f2_fma(W(441), x[11], f2_mul(W(440), x[9])), o[4]); o[5] = f2_fma(p, f2_mul(W(533), x[10]), o[5]); o[6] = f2_fma(p, f2_fma(W(637), x[15], f2_mul(W(636), x[13])), o[6]); o[7] = f2_fma(p, f2_fma(W(725), x[14], f2_mul(W(724), x[12])), o[7]); o[8] = f2_fma(p, f2_fma(W(826), x[15], f2_mul(W(825), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); o[0] = f2_fma(p, f2_fma(W(40), x[14], f2_mul(W(39), x[12])), o[0]); o[1] = f2_fma(p, f2_mul(W(131), x[5]), o[1]); o[2] = f2_fma(p, f2_fma(W(232), x[8], f2_fma(W(231), x[6], W(208))), o[2]); o[3] = f2_fma(p, f2_mul(W(332), x[7]), o[3]); o[4] = f2_fma(p, f2_mul(W(442), x[10]), o[4]); o[5] = f2_fma(p, f2_fma(W(535), x[11], f2_mul(W(534), x[9])), o[5]); o[6] = f2_fma(p, f2_fma(W(639), x[14], f2_mul(W(638), x[12])), o[6]); o[7] = f2_fma(p, f2_fma(W(727), x[15], f2_mul(W(726), x[13])), o[7]); o[8] = f2_fma(p, f2_fma(W(828), x[14], f2_mul(W(827), x[12])), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); o[0] = f2_fma(p, f2_mul(W(41), x[11]), o[0]); o[1] = f2_fma(p, f2_fma(W(133), x[8], f2_fma(W(132), x[6], W(96))), o[1]); o[4] = f2_fma(p, f2_fma(W(444), x[15], f2_mul(W(443), x[13])), o[4]); o[5] = f2_fma(p, f2_fma(W(537), x[14], f2_mul(W(536), x[12])), o[5]); o[6] = f2_fma(p, f2_mul(W(640), x[11]), o[6]); o[7] = f2_fma(p, f2_mul(W(728), x[10]), o[7]); o[8] = f2_fma(p, f2_fma(W(830), x[11], f2_mul(W(829), x[9])), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); o[0] = f2_fma(p, f2_mul(W(42), x[10]), o[0]); o[1] = f2_fma(p, f2_mul(W(134), x[7]), o[1]); o[4] = f2_fma(p, f2_fma(W(446), x[14], f2_mul(W(445), x[12])), o[4]); o[5] = f2_fma(p, f2_fma(W(539), x[15], f2_mul(W(538), x[13])), o[5]); o[6] = f2_fma(p, f2_mul(W(641), x[10]), o[6]); o[7] = f2_fma(p, f2_fma(W(730), x[11], f2_mul(W(729), x[9])), o[7]); o[8] = f2_fma(p, f2_mul(W(831), x[10]), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); o[0] = f2_fma(p, f2_fma(W(44), x[11], f2_mul(W(43), x[9])), o[0]); o[1] = f2_fma(p, f2_fma(W(135), x[8], W(97)), o[1]); o[4] = f2_fma(p, f2_fma(W(448), x[15], f2_mul(W(447), x[13])), o[4]); o[5] = f2_fma(p, f2_fma(W(541), x[14], f2_mul(W(540), x[12])), o[5]); o[6] = f2_fma(p, f2_fma(W(643), x[11], f2_mul(W(642), x[9])), o[6]); o[7] = f2_fma(p, f2_mul(W(731), x[10]), o[7]); o[8] = f2_fma(p, f2_fma(W(833), x[11], f2_mul(W(832), x[9])), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[9]); o[1] = f2_fma(p, f2_fma(W(137), x[11], f2_mul(W(136), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(233), x[14]), o[2]); o[3] = f2_fma(p, f2_mul(W(333), x[13]), o[3]); o[8] = f2_fma(p, W(792), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[10]); o[1] = f2_fma(p, f2_mul(W(138), x[10]), o[1]); o[2] = f2_fma(p, f2_fma(W(235), x[15], f2_mul(W(234), x[13])), o[2]); o[3] = f2_fma(p, f2_mul(W(334), x[12]), o[3]); o[7] = f2_fma(p, W(694), o[7]); } \
      { const unsigned long long p = f2_mul(x[1], x[11]); o[1] = f2_fma(p, f2_mul(W(139), x[11]), o[1]); o[2] = f2_fma(p, f2_fma(W(237), x[14], f2_mul(W(236), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(336), x[15], f2_mul(W(335), x[13])), o[3]); o[6] = f2_fma(p, W(600), o[6]); o[8] = f2_fma(p, W(793), o[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[12]); o[1] = f2_fma(p, f2_fma(W(141), x[14], f2_mul(W(140), x[12])), o[1]); o[5] = f2_fma(p, W(503), o[5]); } \
      { const unsigned long long p = f2_mul(x[1], x[13]); o[1] = f2_fma(p, f2_fma(W(143), x[15], f2_mul(W(142), x[13])), o[1]); o[4] = f2_fma(p, W(413), o[4]); } \
      { const unsigned long long p = f2_mul(x[1], x[14]); o[1] = f2_fma(p, f2_mul(W(144), x[14]), o[1]); o[5] = f2_fma(p, W(504), o[5]); } \
      { const unsigned long long p = f2_mul(x[1], x[15]); o[1] = f2_fma(p, f2_mul(W(145), x[15]), o[1]); o[4] = f2_fma(p, W(414), o[4]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); o[0] = f2_fma(p, f2_fma(W(45), x[6], W(3)), o[0]); o[1] = f2_fma(p, f2_mul(W(146), x[11]), o[1]); o[2] = f2_fma(p, f2_fma(W(239), x[12], f2_mul(W(238), x[2])), o[2]); o[3] = f2_fma(p, f2_fma(W(338), x[13], f2_mul(W(337), x[3])), o[3]); o[4] = f2_fma(p, f2_mul(W(449), x[4]), o[4]); o[5] = f2_fma(p, f2_mul(W(542), x[5]), o[5]); o[6] = f2_fma(p, f2_fma(W(644), x[6], W(601)), o[6]); o[7] = f2_fma(p, f2_mul(W(732), x[7]), o[7]); o[8] = f2_fma(p, f2_mul(W(834), x[8]), o[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); o[0] = f2_fma(p, f2_mul(W(46), x[7]), o[0]); o[1] = f2_fma(p, f2_mul(W(147), x[10]), o[1]); o[2] = f2_fma(p, f2_fma(W(241), x[13], f2_mul(W(240), x[3])), o[2]); o[3] = f2_fma(p, f2_fma(W(340), x[14], f2_mul(W(339), x[12])), o[3]); o[4] = f2_fma(p, f2_mul(W(450), x[5]), o[4]); o[5] = f2_fma(p, f2_mul(W(543), x[4]), o[5]); o[6] = f2_fma(p, f2_mul(W(645), x[7]), o[6]); o[7] = f2_fma(p, f2_fma(W(734), x[8], f2_fma(W(733), x[6], W(695))), o[7]); o[8] = f2_fma(p, f2_mul(W(835), x[7]), o[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); o[0] = f2_fma(p, f2_mul(W(47), x[10]), o[0]); o[1] = f2_fma(p, f2_mul(W(148), x[7]), o[1]); o[2] = f2_fma(p, f2_mul(W(242), x[4]), o[2]); o[3] = f2_fma(p, f2_mul(W(341), x[5]), o[3]); o[4] = f2_fma(p, f2_mul(W(451), x[12]), o[4]); o[5] = f2_fma(p, f2_fma(W(545), x[15], f2_mul(W(544), x[13])), o[5]); o[6] = f2_fma(p, f2_mul(W(646), x[10]), o[6]); o[7] = f2_fma(p, f2_fma(W(736), x[11], f2_mul(W(735), x[9])), o[7]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); o[0] = f2_fma(p, f2_mul(W(48), x[11]), o[0]); o[1] = f2_fma(p, f2_fma(W(150), x[8], f2_fma(W(149), x[6], W(98))), o[1]); o[2] = f2_fma(p, f2_mul(W(243), x[5]), o[2]); o[4] = f2_fma(p, f2_fma(W(453), x[15], f2_mul(W(452), x[13])), o[4]); o[5] = f2_fma(p, f2_fma(W(547), x[14], f2_mul(W(546), x[12])), o[5]); o[6] = f2_fma(p, f2_mul(W(647), x[11]), o[6]); o[7] = f2_fma(p, f2_mul(W(737), x[10]), o[7]); o[8] = f2_fma(p, f2_fma(W(837), x[11], f2_mul(W(836), x[9])), o[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); o[0] = f2_fma(p, f2_mul(W(49), x[12]), o[0]); o[2] = f2_fma(p, f2_fma(W(244), x[6], W(209)), o[2]); o[3] = f2_fma(p, f2_mul(W(342), x[7]), o[3]); o[4] = f2_fma(p, f2_mul(W(454), x[10]), o[4]); o[5] = f2_fma(p, f2_mul(W(548), x[11]), o[5]); o[6] = f2_fma(p, f2_mul(W(648), x[12]), o[6]); o[7] = f2_fma(p, f2_mul(W(738), x[13]), o[7]); o[8] = f2_fma(p, f2_mul(W(838), x[14]), o[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); o[0] = f2_fma(p, f2_mul(W(50), x[13]), o[0]); o[2] = f2_fma(p, f2_mul(W(245), x[7]), o[2]); o[3] = f2_fma(p, f2_fma(W(343), x[8], W(301)), o[3]); o[4] = f2_fma(p, f2_fma(W(456), x[11], f2_mul(W(455), x[9])), o[4]); o[5] = f2_fma(p, f2_mul(W(549), x[10]), o[5]); o[6] = f2_fma(p, f2_mul(W(649), x[13]), o[6]); o[7] = f2_fma(p, f2_fma(W(740), x[14], f2_mul(W(739), x[12])), o[7]); o[8] = f2_fma(p, f2_fma(W(840), x[15], f2_mul(W(839), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); o[0] = f2_fma(p, f2_mul(W(51), x[14]), o[0]); o[2] = f2_fma(p, f2_mul(W(246), x[8]), o[2]); o[5] = f2_fma(p, f2_fma(W(551), x[11], f2_mul(W(550), x[9])), o[5]); o[6] = f2_fma(p, f2_mul(W(650), x[14]), o[6]); o[7] = f2_fma(p, f2_fma(W(742), x[15], f2_mul(W(741), x[13])), o[7]); o[8] = f2_fma(p, f2_mul(W(841), x[12]), o[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[9]); o[1] = f2_fma(p, f2_mul(W(151), x[14]), o[1]); o[2] = f2_fma(p, f2_mul(W(247), x[9]), o[2]); o[3] = f2_fma(p, f2_mul(W(344), x[10]), o[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[10]); o[1] = f2_fma(p, f2_fma(W(153), x[15], f2_mul(W(152), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(248), x[10]), o[2]); o[3] = f2_fma(p, f2_mul(W(345), x[11]), o[3]); o[4] = f2_fma(p, W(415), o[4]); } \
      { const unsigned long long p = f2_mul(x[2], x[11]); o[1] = f2_fma(p, f2_fma(W(155), x[14], f2_mul(W(154), x[12])), o[1]); o[2] = f2_fma(p, f2_mul(W(249), x[11]), o[2]); o[5] = f2_fma(p, W(505), o[5]); } \
      { const unsigned long long p = f2_mul(x[2], x[12]); o[2] = f2_fma(p, f2_mul(W(250), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(346), x[13]), o[3]); o[6] = f2_fma(p, W(602), o[6]); } \
      { const unsigned long long p = f2_mul(x[2], x[13]); o[2] = f2_fma(p, f2_mul(W(251), x[13]), o[2]); o[3] = f2_fma(p, f2_mul(W(347), x[14]), o[3]); o[7] = f2_fma(p, W(696), o[7]); } \
      { const unsigned long long p = f2_mul(x[2], x[14]); o[2] = f2_fma(p, f2_mul(W(252), x[14]), o[2]); o[3] = f2_fma(p, f2_mul(W(348), x[15]), o[3]); o[8] = f2_fma(p, W(794), o[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[15]); o[2] = f2_fma(p, f2_mul(W(253), x[15]), o[2]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); o[0] = f2_fma(p, f2_fma(W(53), x[8], f2_fma(W(52), x[6], W(4))), o[0]); o[1] = f2_fma(p, f2_fma(W(157), x[11], f2_mul(W(156), x[9])), o[1]); o[2] = f2_fma(p, f2_fma(W(255), x[14], f2_mul(W(254), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(351), x[15], f2_fma(W(350), x[13], f2_mul(W(349), x[3]))), o[3]); o[4] = f2_fma(p, f2_mul(W(457), x[4]), o[4]); o[5] = f2_fma(p, f2_mul(W(552), x[5]), o[5]); o[6] = f2_fma(p, f2_fma(W(652), x[8], f2_fma(W(651), x[6], W(603))), o[6]); o[7] = f2_fma(p, f2_mul(W(743), x[7]), o[7]); o[8] = f2_fma(p, f2_fma(W(843), x[8], f2_fma(W(842), x[6], W(795))), o[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); o[0] = f2_fma(p, f2_fma(W(55), x[11], f2_mul(W(54), x[9])), o[0]); o[1] = f2_fma(p, f2_fma(W(158), x[6], W(99)), o[1]); o[2] = f2_fma(p, f2_mul(W(256), x[5]), o[2]); o[3] = f2_fma(p, f2_mul(W(352), x[4]), o[3]); o[4] = f2_fma(p, f2_fma(W(459), x[15], f2_mul(W(458), x[13])), o[4]); o[5] = f2_fma(p, f2_fma(W(554), x[14], f2_mul(W(553), x[12])), o[5]); o[6] = f2_fma(p, f2_fma(W(654), x[11], f2_mul(W(653), x[9])), o[6]); o[7] = f2_fma(p, f2_mul(W(744), x[10]), o[7]); o[8] = f2_fma(p, f2_fma(W(845), x[11], f2_mul(W(844), x[9])), o[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); o[0] = f2_fma(p, f2_mul(W(56), x[10]), o[0]); o[1] = f2_fma(p, f2_mul(W(159), x[7]), o[1]); o[3] = f2_fma(p, f2_mul(W(353), x[5]), o[3]); o[4] = f2_fma(p, f2_fma(W(461), x[14], f2_mul(W(460), x[12])), o[4]); o[5] = f2_fma(p, f2_fma(W(556), x[15], f2_mul(W(555), x[13])), o[5]); o[6] = f2_fma(p, f2_mul(W(655), x[10]), o[6]); o[7] = f2_fma(p, f2_fma(W(746), x[11], f2_mul(W(745), x[9])), o[7]); o[8] = f2_fma(p, f2_mul(W(846), x[10]), o[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); o[0] = f2_fma(p, f2_mul(W(57), x[13]), o[0]); o[2] = f2_fma(p, f2_mul(W(257), x[7]), o[2]); o[3] = f2_fma(p, f2_fma(W(355), x[8], f2_fma(W(354), x[6], W(302))), o[3]); o[4] = f2_fma(p, f2_fma(W(463), x[11], f2_mul(W(462), x[9])), o[4]); o[5] = f2_fma(p, f2_mul(W(557), x[10]), o[5]); o[6] = f2_fma(p, f2_mul(W(656), x[13]), o[6]); o[7] = f2_fma(p, f2_fma(W(748), x[14], f2_mul(W(747), x[12])), o[7]); o[8] = f2_fma(p, f2_fma(W(848), x[15], f2_mul(W(847), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); o[0] = f2_fma(p, f2_fma(W(59), x[14], f2_mul(W(58), x[12])), o[0]); o[2] = f2_fma(p, f2_fma(W(258), x[8], W(210)), o[2]); o[3] = f2_fma(p, f2_mul(W(356), x[7]), o[3]); o[4] = f2_fma(p, f2_mul(W(464), x[10]), o[4]); o[5] = f2_fma(p, f2_fma(W(559), x[11], f2_mul(W(558), x[9])), o[5]); o[6] = f2_fma(p, f2_fma(W(658), x[14], f2_mul(W(657), x[12])), o[6]); o[7] = f2_fma(p, f2_fma(W(750), x[15], f2_mul(W(749), x[13])), o[7]); o[8] = f2_fma(p, f2_fma(W(850), x[14], f2_mul(W(849), x[12])), o[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); o[0] = f2_fma(p, f2_fma(W(61), x[15], f2_mul(W(60), x[13])), o[0]); o[3] = f2_fma(p, f2_fma(W(357), x[8], W(303)), o[3]); o[4] = f2_fma(p, f2_fma(W(466), x[11], f2_mul(W(465), x[9])), o[4]); o[5] = f2_fma(p, f2_mul(W(560), x[10]), o[5]); o[6] = f2_fma(p, f2_fma(W(660), x[15], f2_mul(W(659), x[13])), o[6]); o[7] = f2_fma(p, f2_fma(W(752), x[14], f2_mul(W(751), x[12])), o[7]); o[8] = f2_fma(p, f2_fma(W(852), x[15], f2_mul(W(851), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[9]); o[1] = f2_fma(p, f2_mul(W(160), x[13]), o[1]); o[2] = f2_fma(p, f2_mul(W(259), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(359), x[11], f2_mul(W(358), x[9])), o[3]); o[4] = f2_fma(p, W(416), o[4]); } \
      { const unsigned long long p = f2_mul(x[3], x[10]); o[1] = f2_fma(p, f2_mul(W(161), x[12]), o[1]); o[2] = f2_fma(p, f2_mul(W(260), x[11]), o[2]); o[3] = f2_fma(p, f2_mul(W(360), x[10]), o[3]); o[5] = f2_fma(p, W(506), o[5]); } \
      { const unsigned long long p = f2_mul(x[3], x[11]); o[1] = f2_fma(p, f2_fma(W(163), x[15], f2_mul(W(162), x[13])), o[1]); o[3] = f2_fma(p, f2_mul(W(361), x[11]), o[3]); o[4] = f2_fma(p, W(417), o[4]); } \
      { const unsigned long long p = f2_mul(x[3], x[12]); o[2] = f2_fma(p, f2_mul(W(261), x[13]), o[2]); o[3] = f2_fma(p, f2_fma(W(363), x[14], f2_mul(W(362), x[12])), o[3]); o[7] = f2_fma(p, W(697), o[7]); } \
      { const unsigned long long p = f2_mul(x[3], x[13]); o[2] = f2_fma(p, f2_mul(W(262), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(365), x[15], f2_mul(W(364), x[13])), o[3]); o[6] = f2_fma(p, W(604), o[6]); o[8] = f2_fma(p, W(796), o[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[14]); o[2] = f2_fma(p, f2_mul(W(263), x[15]), o[2]); o[3] = f2_fma(p, f2_mul(W(366), x[14]), o[3]); o[7] = f2_fma(p, W(698), o[7]); } \
      { const unsigned long long p = f2_mul(x[3], x[15]); o[3] = f2_fma(p, f2_mul(W(367), x[15]), o[3]); o[8] = f2_fma(p, W(797), o[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); o[0] = f2_fma(p, f2_fma(W(62), x[6], W(5)), o[0]); o[1] = f2_fma(p, f2_fma(W(165), x[11], f2_mul(W(164), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(264), x[12]), o[2]); o[3] = f2_fma(p, f2_fma(W(369), x[15], f2_mul(W(368), x[13])), o[3]); o[4] = f2_fma(p, f2_mul(W(467), x[4]), o[4]); o[5] = f2_fma(p, f2_mul(W(561), x[5]), o[5]); o[6] = f2_fma(p, f2_fma(W(661), x[6], W(605)), o[6]); o[7] = f2_fma(p, f2_mul(W(753), x[7]), o[7]); o[8] = f2_fma(p, f2_mul(W(853), x[8]), o[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); o[0] = f2_fma(p, f2_mul(W(63), x[7]), o[0]); o[1] = f2_fma(p, f2_mul(W(166), x[10]), o[1]); o[2] = f2_fma(p, f2_fma(W(266), x[15], f2_mul(W(265), x[13])), o[2]); o[3] = f2_fma(p, f2_fma(W(371), x[14], f2_mul(W(370), x[12])), o[3]); o[4] = f2_fma(p, f2_mul(W(468), x[5]), o[4]); o[7] = f2_fma(p, W(699), o[7]); } \
      { const unsigned long long p = f2_mul(x[4], x[6]); o[1] = f2_fma(p, f2_fma(W(168), x[15], f2_mul(W(167), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(267), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(373), x[11], f2_mul(W(372), x[9])), o[3]); o[4] = f2_fma(p, f2_fma(W(469), x[6], W(418)), o[4]); } \
      { const unsigned long long p = f2_mul(x[4], x[7]); o[1] = f2_fma(p, f2_fma(W(170), x[14], f2_mul(W(169), x[12])), o[1]); o[2] = f2_fma(p, f2_fma(W(269), x[11], f2_mul(W(268), x[9])), o[2]); o[3] = f2_fma(p, f2_mul(W(374), x[10]), o[3]); o[4] = f2_fma(p, f2_mul(W(470), x[7]), o[4]); o[5] = f2_fma(p, W(507), o[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[8]); o[1] = f2_fma(p, f2_mul(W(171), x[15]), o[1]); o[3] = f2_fma(p, f2_mul(W(375), x[9]), o[3]); o[4] = f2_fma(p, f2_mul(W(471), x[8]), o[4]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); o[0] = f2_fma(p, f2_mul(W(64), x[13]), o[0]); o[3] = f2_fma(p, W(304), o[3]); o[4] = f2_fma(p, f2_fma(W(473), x[11], f2_mul(W(472), x[9])), o[4]); o[5] = f2_fma(p, f2_mul(W(562), x[10]), o[5]); o[6] = f2_fma(p, f2_mul(W(662), x[13]), o[6]); o[7] = f2_fma(p, f2_fma(W(755), x[14], f2_mul(W(754), x[12])), o[7]); o[8] = f2_fma(p, f2_mul(W(854), x[13]), o[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); o[0] = f2_fma(p, f2_mul(W(65), x[12]), o[0]); o[2] = f2_fma(p, W(211), o[2]); o[4] = f2_fma(p, f2_mul(W(474), x[10]), o[4]); o[5] = f2_fma(p, f2_mul(W(563), x[11]), o[5]); o[6] = f2_fma(p, f2_mul(W(663), x[12]), o[6]); o[7] = f2_fma(p, f2_fma(W(757), x[15], f2_mul(W(756), x[13])), o[7]); o[8] = f2_fma(p, f2_mul(W(855), x[14]), o[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); o[0] = f2_fma(p, f2_fma(W(67), x[15], f2_mul(W(66), x[13])), o[0]); o[3] = f2_fma(p, W(305), o[3]); o[4] = f2_fma(p, f2_mul(W(475), x[11]), o[4]); o[6] = f2_fma(p, f2_fma(W(665), x[15], f2_mul(W(664), x[13])), o[6]); o[7] = f2_fma(p, f2_fma(W(759), x[14], f2_mul(W(758), x[12])), o[7]); o[8] = f2_fma(p, f2_mul(W(856), x[15]), o[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[12]); o[4] = f2_fma(p, f2_mul(W(476), x[12]), o[4]); o[5] = f2_fma(p, f2_fma(W(565), x[15], f2_mul(W(564), x[13])), o[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[13]); o[1] = f2_fma(p, W(100), o[1]); o[4] = f2_fma(p, f2_fma(W(478), x[15], f2_mul(W(477), x[13])), o[4]); o[5] = f2_fma(p, f2_mul(W(566), x[14]), o[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[14]); o[4] = f2_fma(p, f2_mul(W(479), x[14]), o[4]); o[5] = f2_fma(p, f2_mul(W(567), x[15]), o[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[15]); o[1] = f2_fma(p, W(101), o[1]); o[4] = f2_fma(p, f2_mul(W(480), x[15]), o[4]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); o[0] = f2_fma(p, f2_fma(W(69), x[8], f2_fma(W(68), x[6], W(6))), o[0]); o[1] = f2_fma(p, f2_fma(W(173), x[11], f2_mul(W(172), x[9])), o[1]); o[2] = f2_fma(p, f2_fma(W(271), x[14], f2_mul(W(270), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(377), x[15], f2_mul(W(376), x[13])), o[3]); o[5] = f2_fma(p, f2_mul(W(568), x[5]), o[5]); o[6] = f2_fma(p, f2_fma(W(666), x[6], W(606)), o[6]); o[7] = f2_fma(p, f2_mul(W(760), x[7]), o[7]); o[8] = f2_fma(p, f2_fma(W(857), x[8], W(798)), o[8]); } \
      { const unsigned long long p = f2_mul(x[5], x[6]); o[1] = f2_fma(p, f2_fma(W(175), x[14], f2_mul(W(174), x[12])), o[1]); o[2] = f2_fma(p, f2_mul(W(272), x[11]), o[2]); o[3] = f2_fma(p, f2_mul(W(378), x[10]), o[3]); o[5] = f2_fma(p, f2_fma(W(569), x[6], W(508)), o[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[7]); o[1] = f2_fma(p, f2_fma(W(177), x[15], f2_mul(W(176), x[13])), o[1]); o[2] = f2_fma(p, f2_mul(W(273), x[10]), o[2]); o[3] = f2_fma(p, f2_fma(W(380), x[11], f2_mul(W(379), x[9])), o[3]); o[4] = f2_fma(p, W(419), o[4]); o[5] = f2_fma(p, f2_mul(W(570), x[7]), o[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[8]); o[1] = f2_fma(p, f2_fma(W(179), x[14], f2_mul(W(178), x[12])), o[1]); o[2] = f2_fma(p, f2_fma(W(275), x[11], f2_mul(W(274), x[9])), o[2]); o[3] = f2_fma(p, f2_mul(W(381), x[10]), o[3]); o[5] = f2_fma(p, f2_fma(W(571), x[8], W(509)), o[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); o[0] = f2_fma(p, f2_mul(W(70), x[14]), o[0]); o[4] = f2_fma(p, f2_mul(W(481), x[10]), o[4]); o[5] = f2_fma(p, f2_fma(W(573), x[11], f2_mul(W(572), x[9])), o[5]); o[6] = f2_fma(p, f2_mul(W(667), x[14]), o[6]); o[7] = f2_fma(p, f2_mul(W(761), x[13]), o[7]); o[8] = f2_fma(p, f2_fma(W(859), x[14], f2_mul(W(858), x[12])), o[8]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); o[0] = f2_fma(p, f2_fma(W(72), x[15], f2_mul(W(71), x[13])), o[0]); o[3] = f2_fma(p, W(306), o[3]); o[4] = f2_fma(p, f2_mul(W(482), x[11]), o[4]); o[5] = f2_fma(p, f2_mul(W(574), x[10]), o[5]); o[6] = f2_fma(p, f2_fma(W(669), x[15], f2_mul(W(668), x[13])), o[6]); o[7] = f2_fma(p, f2_mul(W(762), x[12]), o[7]); o[8] = f2_fma(p, f2_fma(W(861), x[15], f2_mul(W(860), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); o[0] = f2_fma(p, f2_fma(W(74), x[14], f2_mul(W(73), x[12])), o[0]); o[2] = f2_fma(p, W(212), o[2]); o[5] = f2_fma(p, f2_mul(W(575), x[11]), o[5]); o[6] = f2_fma(p, f2_fma(W(671), x[14], f2_mul(W(670), x[12])), o[6]); o[7] = f2_fma(p, f2_fma(W(764), x[15], f2_mul(W(763), x[13])), o[7]); o[8] = f2_fma(p, f2_fma(W(863), x[14], f2_mul(W(862), x[12])), o[8]); } \
      { const unsigned long long p = f2_mul(x[5], x[12]); o[1] = f2_fma(p, W(102), o[1]); o[4] = f2_fma(p, f2_fma(W(484), x[15], f2_mul(W(483), x[13])), o[4]); o[5] = f2_fma(p, f2_fma(W(577), x[14], f2_mul(W(576), x[12])), o[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[13]); o[4] = f2_fma(p, f2_mul(W(485), x[14]), o[4]); o[5] = f2_fma(p, f2_fma(W(579), x[15], f2_mul(W(578), x[13])), o[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[14]); o[1] = f2_fma(p, W(103), o[1]); o[4] = f2_fma(p, f2_mul(W(486), x[15]), o[4]); o[5] = f2_fma(p, f2_mul(W(580), x[14]), o[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[15]); o[5] = f2_fma(p, f2_mul(W(581), x[15]), o[5]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); o[0] = f2_fma(p, f2_fma(W(75), x[6], W(7)), o[0]); o[1] = f2_fma(p, f2_mul(W(180), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(276), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(382), x[13]), o[3]); o[6] = f2_fma(p, f2_fma(W(672), x[6], W(607)), o[6]); o[7] = f2_fma(p, f2_mul(W(765), x[7]), o[7]); o[8] = f2_fma(p, f2_mul(W(864), x[8]), o[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); o[0] = f2_fma(p, f2_mul(W(76), x[7]), o[0]); o[1] = f2_fma(p, f2_mul(W(181), x[10]), o[1]); o[2] = f2_fma(p, f2_mul(W(277), x[13]), o[2]); o[3] = f2_fma(p, f2_fma(W(384), x[14], f2_mul(W(383), x[12])), o[3]); o[6] = f2_fma(p, f2_mul(W(673), x[7]), o[6]); o[7] = f2_fma(p, W(700), o[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); o[0] = f2_fma(p, f2_mul(W(77), x[8]), o[0]); o[1] = f2_fma(p, f2_fma(W(183), x[11], f2_mul(W(182), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(278), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(386), x[15], f2_mul(W(385), x[13])), o[3]); o[6] = f2_fma(p, f2_mul(W(674), x[8]), o[6]); o[8] = f2_fma(p, W(799), o[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); o[0] = f2_fma(p, f2_mul(W(78), x[9]), o[0]); o[4] = f2_fma(p, f2_mul(W(487), x[13]), o[4]); o[5] = f2_fma(p, f2_mul(W(582), x[14]), o[5]); o[6] = f2_fma(p, f2_mul(W(675), x[9]), o[6]); o[7] = f2_fma(p, f2_mul(W(766), x[10]), o[7]); o[8] = f2_fma(p, f2_mul(W(865), x[11]), o[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[10]); o[4] = f2_fma(p, f2_mul(W(488), x[12]), o[4]); o[5] = f2_fma(p, f2_fma(W(584), x[15], f2_mul(W(583), x[13])), o[5]); o[6] = f2_fma(p, f2_mul(W(676), x[10]), o[6]); o[7] = f2_fma(p, f2_mul(W(767), x[11]), o[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); o[0] = f2_fma(p, f2_mul(W(79), x[11]), o[0]); o[1] = f2_fma(p, W(104), o[1]); o[4] = f2_fma(p, f2_fma(W(490), x[15], f2_mul(W(489), x[13])), o[4]); o[5] = f2_fma(p, f2_fma(W(586), x[14], f2_mul(W(585), x[12])), o[5]); o[6] = f2_fma(p, f2_mul(W(677), x[11]), o[6]); o[8] = f2_fma(p, f2_mul(W(866), x[11]), o[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); o[0] = f2_fma(p, f2_mul(W(80), x[12]), o[0]); o[2] = f2_fma(p, W(213), o[2]); o[6] = f2_fma(p, f2_mul(W(678), x[12]), o[6]); o[7] = f2_fma(p, f2_mul(W(768), x[13]), o[7]); o[8] = f2_fma(p, f2_mul(W(867), x[14]), o[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); o[0] = f2_fma(p, f2_mul(W(81), x[13]), o[0]); o[3] = f2_fma(p, W(307), o[3]); o[6] = f2_fma(p, f2_mul(W(679), x[13]), o[6]); o[7] = f2_fma(p, f2_mul(W(769), x[14]), o[7]); o[8] = f2_fma(p, f2_fma(W(869), x[15], f2_mul(W(868), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[14]); o[6] = f2_fma(p, f2_mul(W(680), x[14]), o[6]); o[7] = f2_fma(p, f2_mul(W(770), x[15]), o[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); o[0] = f2_fma(p, f2_mul(W(82), x[15]), o[0]); o[6] = f2_fma(p, f2_mul(W(681), x[15]), o[6]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); o[0] = f2_fma(p, f2_fma(W(83), x[8], W(8)), o[0]); o[1] = f2_fma(p, f2_fma(W(185), x[11], f2_mul(W(184), x[9])), o[1]); o[2] = f2_fma(p, f2_fma(W(280), x[14], f2_mul(W(279), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(388), x[15], f2_mul(W(387), x[13])), o[3]); o[6] = f2_fma(p, W(608), o[6]); o[7] = f2_fma(p, f2_mul(W(771), x[7]), o[7]); o[8] = f2_fma(p, f2_fma(W(870), x[8], W(800)), o[8]); } \
      { const unsigned long long p = f2_mul(x[7], x[8]); o[1] = f2_fma(p, f2_mul(W(186), x[10]), o[1]); o[2] = f2_fma(p, f2_fma(W(282), x[15], f2_mul(W(281), x[13])), o[2]); o[3] = f2_fma(p, f2_fma(W(390), x[14], f2_mul(W(389), x[12])), o[3]); o[7] = f2_fma(p, f2_fma(W(772), x[8], W(701)), o[7]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); o[0] = f2_fma(p, f2_mul(W(84), x[10]), o[0]); o[4] = f2_fma(p, f2_fma(W(492), x[14], f2_mul(W(491), x[12])), o[4]); o[5] = f2_fma(p, f2_mul(W(587), x[13]), o[5]); o[6] = f2_fma(p, f2_mul(W(682), x[10]), o[6]); o[7] = f2_fma(p, f2_fma(W(774), x[11], f2_mul(W(773), x[9])), o[7]); o[8] = f2_fma(p, f2_mul(W(871), x[10]), o[8]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); o[0] = f2_fma(p, f2_mul(W(85), x[11]), o[0]); o[1] = f2_fma(p, W(105), o[1]); o[4] = f2_fma(p, f2_fma(W(494), x[15], f2_mul(W(493), x[13])), o[4]); o[5] = f2_fma(p, f2_mul(W(588), x[12]), o[5]); o[6] = f2_fma(p, f2_mul(W(683), x[11]), o[6]); o[7] = f2_fma(p, f2_mul(W(775), x[10]), o[7]); o[8] = f2_fma(p, f2_mul(W(872), x[11]), o[8]); } \
      { const unsigned long long p = f2_mul(x[7], x[11]); o[4] = f2_fma(p, f2_fma(W(496), x[14], f2_mul(W(495), x[12])), o[4]); o[5] = f2_fma(p, f2_fma(W(590), x[15], f2_mul(W(589), x[13])), o[5]); o[7] = f2_fma(p, f2_mul(W(776), x[11]), o[7]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); o[0] = f2_fma(p, f2_mul(W(86), x[13]), o[0]); o[3] = f2_fma(p, W(308), o[3]); o[6] = f2_fma(p, f2_mul(W(684), x[13]), o[6]); o[7] = f2_fma(p, f2_fma(W(778), x[14], f2_mul(W(777), x[12])), o[7]); o[8] = f2_fma(p, f2_fma(W(874), x[15], f2_mul(W(873), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); o[0] = f2_fma(p, f2_mul(W(87), x[14]), o[0]); o[2] = f2_fma(p, W(214), o[2]); o[6] = f2_fma(p, f2_mul(W(685), x[14]), o[6]); o[7] = f2_fma(p, f2_fma(W(780), x[15], f2_mul(W(779), x[13])), o[7]); o[8] = f2_fma(p, f2_mul(W(875), x[14]), o[8]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); o[0] = f2_fma(p, f2_mul(W(88), x[15]), o[0]); o[3] = f2_fma(p, W(309), o[3]); o[6] = f2_fma(p, f2_mul(W(686), x[15]), o[6]); o[7] = f2_fma(p, f2_mul(W(781), x[14]), o[7]); o[8] = f2_fma(p, f2_mul(W(876), x[15]), o[8]); } \
      { const unsigned long long p = f2_mul(x[7], x[15]); o[7] = f2_fma(p, f2_mul(W(782), x[15]), o[7]); } \
      { const unsigned long long p = f2_mul(x[8], x[8]); o[0] = f2_fma(p, W(9), o[0]); o[1] = f2_fma(p, f2_fma(W(188), x[11], f2_mul(W(187), x[9])), o[1]); o[2] = f2_fma(p, f2_mul(W(283), x[12]), o[2]); o[3] = f2_fma(p, f2_fma(W(392), x[15], f2_mul(W(391), x[13])), o[3]); o[6] = f2_fma(p, W(609), o[6]); o[8] = f2_fma(p, f2_mul(W(877), x[8]), o[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); o[0] = f2_fma(p, f2_mul(W(89), x[11]), o[0]); o[1] = f2_fma(p, W(106), o[1]); o[4] = f2_fma(p, f2_mul(W(497), x[13]), o[4]); o[5] = f2_fma(p, f2_fma(W(592), x[14], f2_mul(W(591), x[12])), o[5]); o[6] = f2_fma(p, f2_mul(W(687), x[11]), o[6]); o[7] = f2_fma(p, f2_mul(W(783), x[10]), o[7]); o[8] = f2_fma(p, f2_fma(W(879), x[11], f2_mul(W(878), x[9])), o[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[10]); o[4] = f2_fma(p, f2_mul(W(498), x[14]), o[4]); o[5] = f2_fma(p, f2_fma(W(594), x[15], f2_mul(W(593), x[13])), o[5]); o[7] = f2_fma(p, f2_mul(W(784), x[11]), o[7]); o[8] = f2_fma(p, f2_mul(W(880), x[10]), o[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); o[0] = f2_fma(p, f2_mul(W(90), x[11]), o[0]); o[1] = f2_fma(p, W(107), o[1]); o[4] = f2_fma(p, f2_mul(W(499), x[15]), o[4]); o[5] = f2_fma(p, f2_fma(W(596), x[14], f2_mul(W(595), x[12])), o[5]); o[6] = f2_fma(p, f2_mul(W(688), x[11]), o[6]); o[8] = f2_fma(p, f2_mul(W(881), x[11]), o[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); o[0] = f2_fma(p, f2_mul(W(91), x[14]), o[0]); o[6] = f2_fma(p, f2_mul(W(689), x[14]), o[6]); o[7] = f2_fma(p, f2_fma(W(786), x[15], f2_mul(W(785), x[13])), o[7]); o[8] = f2_fma(p, f2_mul(W(882), x[12]), o[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); o[0] = f2_fma(p, f2_fma(W(93), x[15], f2_mul(W(92), x[13])), o[0]); o[3] = f2_fma(p, W(310), o[3]); o[6] = f2_fma(p, f2_fma(W(691), x[15], f2_mul(W(690), x[13])), o[6]); o[7] = f2_fma(p, f2_mul(W(787), x[14]), o[7]); o[8] = f2_fma(p, f2_fma(W(884), x[15], f2_mul(W(883), x[13])), o[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[14]); o[2] = f2_fma(p, W(215), o[2]); o[7] = f2_fma(p, f2_mul(W(788), x[15]), o[7]); o[8] = f2_fma(p, f2_mul(W(885), x[14]), o[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[15]); o[3] = f2_fma(p, W(311), o[3]); o[8] = f2_fma(p, f2_mul(W(886), x[15]), o[8]); } \
      { const unsigned long long p = f2_mul(x[9], x[9]); o[0] = f2_fma(p, W(10), o[0]); o[1] = f2_fma(p, f2_mul(W(189), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(284), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(393), x[13]), o[3]); o[6] = f2_fma(p, W(610), o[6]); } \
      { const unsigned long long p = f2_mul(x[9], x[10]); o[1] = f2_fma(p, f2_mul(W(190), x[10]), o[1]); o[2] = f2_fma(p, f2_mul(W(285), x[13]), o[2]); o[3] = f2_fma(p, f2_fma(W(395), x[14], f2_mul(W(394), x[12])), o[3]); o[7] = f2_fma(p, W(702), o[7]); } \
      { const unsigned long long p = f2_mul(x[9], x[11]); o[1] = f2_fma(p, f2_mul(W(191), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(286), x[14]), o[2]); o[3] = f2_fma(p, f2_mul(W(396), x[13]), o[3]); o[8] = f2_fma(p, W(801), o[8]); } \
      { const unsigned long long p = f2_mul(x[9], x[12]); o[1] = f2_fma(p, f2_mul(W(192), x[14]), o[1]); } \
      { const unsigned long long p = f2_mul(x[9], x[13]); o[1] = f2_fma(p, f2_mul(W(193), x[13]), o[1]); o[4] = f2_fma(p, W(420), o[4]); } \
      { const unsigned long long p = f2_mul(x[9], x[14]); o[1] = f2_fma(p, f2_mul(W(194), x[14]), o[1]); o[5] = f2_fma(p, W(510), o[5]); } \
      { const unsigned long long p = f2_mul(x[10], x[10]); o[0] = f2_fma(p, W(11), o[0]); o[1] = f2_fma(p, f2_mul(W(195), x[11]), o[1]); o[2] = f2_fma(p, f2_mul(W(287), x[12]), o[2]); o[3] = f2_fma(p, f2_fma(W(398), x[15], f2_mul(W(397), x[13])), o[3]); } \
      { const unsigned long long p = f2_mul(x[10], x[11]); o[2] = f2_fma(p, f2_fma(W(289), x[15], f2_mul(W(288), x[13])), o[2]); o[3] = f2_fma(p, f2_mul(W(399), x[12]), o[3]); o[7] = f2_fma(p, W(703), o[7]); } \
      { const unsigned long long p = f2_mul(x[10], x[12]); o[1] = f2_fma(p, f2_fma(W(197), x[15], f2_mul(W(196), x[13])), o[1]); o[4] = f2_fma(p, W(421), o[4]); } \
      { const unsigned long long p = f2_mul(x[10], x[13]); o[5] = f2_fma(p, W(511), o[5]); } \
      { const unsigned long long p = f2_mul(x[10], x[14]); o[1] = f2_fma(p, f2_mul(W(198), x[15]), o[1]); } \
      { const unsigned long long p = f2_mul(x[10], x[15]); o[5] = f2_fma(p, W(512), o[5]); } \
      { const unsigned long long p = f2_mul(x[11], x[11]); o[0] = f2_fma(p, W(12), o[0]); o[1] = f2_fma(p, f2_mul(W(199), x[11]), o[1]); o[2] = f2_fma(p, f2_fma(W(291), x[14], f2_mul(W(290), x[12])), o[2]); o[3] = f2_fma(p, f2_fma(W(401), x[15], f2_mul(W(400), x[13])), o[3]); o[6] = f2_fma(p, W(611), o[6]); o[8] = f2_fma(p, W(802), o[8]); } \
      { const unsigned long long p = f2_mul(x[11], x[12]); o[1] = f2_fma(p, f2_fma(W(201), x[14], f2_mul(W(200), x[12])), o[1]); o[5] = f2_fma(p, W(513), o[5]); } \
      { const unsigned long long p = f2_mul(x[11], x[13]); o[1] = f2_fma(p, f2_fma(W(203), x[15], f2_mul(W(202), x[13])), o[1]); o[4] = f2_fma(p, W(422), o[4]); } \
      { const unsigned long long p = f2_mul(x[11], x[14]); o[1] = f2_fma(p, f2_mul(W(204), x[14]), o[1]); o[5] = f2_fma(p, W(514), o[5]); } \
      { const unsigned long long p = f2_mul(x[11], x[15]); o[1] = f2_fma(p, f2_mul(W(205), x[15]), o[1]); o[4] = f2_fma(p, W(423), o[4]); } \
      { const unsigned long long p = f2_mul(x[12], x[12]); o[0] = f2_fma(p, W(13), o[0]); o[2] = f2_fma(p, f2_mul(W(292), x[12]), o[2]); o[3] = f2_fma(p, f2_mul(W(402), x[13]), o[3]); o[6] = f2_fma(p, W(612), o[6]); } \
      { const unsigned long long p = f2_mul(x[12], x[13]); o[2] = f2_fma(p, f2_mul(W(293), x[13]), o[2]); o[3] = f2_fma(p, f2_mul(W(403), x[14]), o[3]); o[7] = f2_fma(p, W(704), o[7]); } \
      { const unsigned long long p = f2_mul(x[12], x[14]); o[2] = f2_fma(p, f2_mul(W(294), x[14]), o[2]); o[3] = f2_fma(p, f2_mul(W(404), x[15]), o[3]); o[8] = f2_fma(p, W(803), o[8]); } \
      { const unsigned long long p = f2_mul(x[12], x[15]); o[2] = f2_fma(p, f2_mul(W(295), x[15]), o[2]); } \
      { const unsigned long long p = f2_mul(x[13], x[13]); o[0] = f2_fma(p, W(14), o[0]); o[2] = f2_fma(p, f2_mul(W(296), x[14]), o[2]); o[3] = f2_fma(p, f2_fma(W(406), x[15], f2_mul(W(405), x[13])), o[3]); o[6] = f2_fma(p, W(613), o[6]); o[8] = f2_fma(p, W(804), o[8]); } \
      { const unsigned long long p = f2_mul(x[13], x[14]); o[2] = f2_fma(p, f2_mul(W(297), x[15]), o[2]); o[3] = f2_fma(p, f2_mul(W(407), x[14]), o[3]); o[7] = f2_fma(p, W(705), o[7]); } \
      { const unsigned long long p = f2_mul(x[13], x[15]); o[3] = f2_fma(p, f2_mul(W(408), x[15]), o[3]); o[8] = f2_fma(p, W(805), o[8]); } \
      { const unsigned long long p = f2_mul(x[14], x[14]); o[0] = f2_fma(p, W(15), o[0]); o[3] = f2_fma(p, f2_mul(W(409), x[15]), o[3]); } \
      { const unsigned long long p = f2_mul(x[14], x[15]); o[7] = f2_fma(p, W(706), o[7]); } \
      { const unsigned long long p = f2_mul(x[15], x[15]); o[0] = f2_fma(p, W(16), o[0]); o[6] = f2_fma(p, W(614), o[6]); }
#define SXB_S2_M0_REVERSE_BODY \
      g[0] = f2_fma(W(0), adj[0], g[0]); \
      g[1] = f2_fma(W(94), adj[1], g[1]); \
      g[2] = f2_fma(W(206), adj[2], g[2]); \
      g[3] = f2_fma(W(298), adj[3], g[3]); \
      g[4] = f2_fma(W(410), adj[4], g[4]); \
      g[5] = f2_fma(W(500), adj[5], g[5]); \
      g[6] = f2_fma(W(597), adj[6], g[6]); \
      g[7] = f2_fma(W(692), adj[7], g[7]); \
      g[8] = f2_fma(W(789), adj[8], g[8]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); unsigned long long v; v = f2_mul(W(1), adj[0]); { const unsigned long long s = f2_mul(W(17), adj[0]); g[0] = f2_fma(s, p, g[0]); v = f2_fma(s, x[0], v); } { const unsigned long long s = f2_mul(W(108), adj[1]); g[1] = f2_fma(s, p, g[1]); v = f2_fma(s, x[1], v); } { const unsigned long long s = f2_mul(W(216), adj[2]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(312), adj[3]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(424), adj[4]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(515), adj[5]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(615), adj[6]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(707), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(806), adj[8]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[0] = f2_fma(v, x[0], g[0]); g[0] = f2_fma(v, x[0], g[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); unsigned long long v; v = f2_mul(W(95), adj[1]); { const unsigned long long s = f2_fma(W(807), adj[8], f2_fma(W(616), adj[6], f2_mul(W(18), adj[0]))); g[1] = f2_fma(s, p, g[1]); v = f2_fma(s, x[1], v); } { const unsigned long long s = f2_mul(W(516), adj[5]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(425), adj[4]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(313), adj[3]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(217), adj[2]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(109), adj[1]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(110), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(808), adj[8]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(708), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_fma(W(809), adj[8], f2_mul(W(617), adj[6])); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(517), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(426), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(518), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(427), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[1], g[0]); g[1] = f2_fma(v, x[0], g[1]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); unsigned long long v; v = f2_mul(W(207), adj[2]); { const unsigned long long s = f2_fma(W(618), adj[6], f2_mul(W(19), adj[0])); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(709), adj[7]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(111), adj[1]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(218), adj[2]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(314), adj[3]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(428), adj[4]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(519), adj[5]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(619), adj[6]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(710), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(810), adj[8]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[0] = f2_fma(v, x[2], g[0]); g[2] = f2_fma(v, x[0], g[2]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); unsigned long long v; v = f2_mul(W(299), adj[3]); { const unsigned long long s = f2_fma(W(811), adj[8], f2_fma(W(620), adj[6], f2_mul(W(20), adj[0]))); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(112), adj[1]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(315), adj[3]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(219), adj[2]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(316), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(429), adj[4]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(520), adj[5]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(430), adj[4]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(711), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(812), adj[8], f2_mul(W(621), adj[6])); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(712), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(813), adj[8]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[3], g[0]); g[3] = f2_fma(v, x[0], g[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); unsigned long long v; v = f2_mul(W(411), adj[4]); { const unsigned long long s = f2_fma(W(622), adj[6], f2_mul(W(21), adj[0])); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(713), adj[7]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(431), adj[4]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(521), adj[5]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(317), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(220), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(318), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(113), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(114), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[4], g[0]); g[4] = f2_fma(v, x[0], g[4]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); unsigned long long v; v = f2_mul(W(501), adj[5]); { const unsigned long long s = f2_fma(W(814), adj[8], f2_fma(W(623), adj[6], f2_mul(W(22), adj[0]))); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(522), adj[5]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(432), adj[4]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(523), adj[5]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(319), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(221), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(115), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(116), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[0] = f2_fma(v, x[5], g[0]); g[5] = f2_fma(v, x[0], g[5]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); unsigned long long v; v = f2_mul(W(598), adj[6]); { const unsigned long long s = f2_fma(W(624), adj[6], f2_mul(W(23), adj[0])); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(714), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(815), adj[8]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(117), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(222), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(320), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[0] = f2_fma(v, x[6], g[0]); g[6] = f2_fma(v, x[0], g[6]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); unsigned long long v; v = f2_mul(W(693), adj[7]); { const unsigned long long s = f2_fma(W(816), adj[8], f2_fma(W(625), adj[6], f2_mul(W(24), adj[0]))); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(715), adj[7]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(118), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(321), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(223), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(322), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[0] = f2_fma(v, x[7], g[0]); g[7] = f2_fma(v, x[0], g[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); unsigned long long v; v = f2_mul(W(790), adj[8]); { const unsigned long long s = f2_fma(W(626), adj[6], f2_mul(W(25), adj[0])); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(119), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(120), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(323), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(224), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(324), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[8], g[0]); g[8] = f2_fma(v, x[0], g[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); unsigned long long v; { const unsigned long long s = f2_fma(W(627), adj[6], f2_mul(W(26), adj[0])); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(716), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(817), adj[8]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(433), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(524), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[0] = f2_fma(v, x[9], g[0]); g[9] = f2_fma(v, x[0], g[9]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(27), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(717), adj[7]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(434), adj[4]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(525), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(526), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[10], g[0]); g[10] = f2_fma(v, x[0], g[10]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); unsigned long long v; { const unsigned long long s = f2_fma(W(818), adj[8], f2_fma(W(628), adj[6], f2_mul(W(28), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } { const unsigned long long s = f2_mul(W(527), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(435), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(528), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(436), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[11], g[0]); g[11] = f2_fma(v, x[0], g[11]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); unsigned long long v; { const unsigned long long s = f2_fma(W(629), adj[6], f2_mul(W(29), adj[0])); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(718), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(819), adj[8]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[0] = f2_fma(v, x[12], g[0]); g[12] = f2_fma(v, x[0], g[12]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); unsigned long long v; { const unsigned long long s = f2_fma(W(820), adj[8], f2_fma(W(630), adj[6], f2_mul(W(30), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(719), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(821), adj[8]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[13], g[0]); g[13] = f2_fma(v, x[0], g[13]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(31), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } { const unsigned long long s = f2_mul(W(720), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[0] = f2_fma(v, x[14], g[0]); g[14] = f2_fma(v, x[0], g[14]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); unsigned long long v; { const unsigned long long s = f2_fma(W(631), adj[6], f2_mul(W(32), adj[0])); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[0] = f2_fma(v, x[15], g[0]); g[15] = f2_fma(v, x[0], g[15]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); unsigned long long v; v = f2_fma(W(791), adj[8], f2_fma(W(599), adj[6], f2_mul(W(2), adj[0]))); { const unsigned long long s = f2_mul(W(121), adj[1]); g[1] = f2_fma(s, p, g[1]); v = f2_fma(s, x[1], v); } { const unsigned long long s = f2_mul(W(225), adj[2]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(325), adj[3]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(437), adj[4]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(529), adj[5]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_fma(W(822), adj[8], f2_fma(W(632), adj[6], f2_mul(W(33), adj[0]))); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(721), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_fma(W(823), adj[8], f2_fma(W(633), adj[6], f2_mul(W(34), adj[0]))); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(122), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(123), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(226), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(326), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(227), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(327), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[1], g[1]); g[1] = f2_fma(v, x[1], g[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); unsigned long long v; v = f2_mul(W(502), adj[5]); { const unsigned long long s = f2_mul(W(124), adj[1]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(722), adj[7]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_fma(W(824), adj[8], f2_fma(W(634), adj[6], f2_mul(W(35), adj[0]))); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(530), adj[5]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(438), adj[4]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(531), adj[5]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(328), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(228), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(125), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(126), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[2], g[1]); g[2] = f2_fma(v, x[1], g[2]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); unsigned long long v; v = f2_mul(W(412), adj[4]); { const unsigned long long s = f2_mul(W(127), adj[1]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_fma(W(635), adj[6], f2_mul(W(36), adj[0])); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(723), adj[7]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(439), adj[4]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(532), adj[5]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(329), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(229), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(330), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(128), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(129), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[3], g[1]); g[3] = f2_fma(v, x[1], g[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); unsigned long long v; v = f2_mul(W(300), adj[3]); { const unsigned long long s = f2_mul(W(130), adj[1]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(331), adj[3]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(230), adj[2]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(440), adj[4]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(533), adj[5]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(441), adj[4]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(724), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(825), adj[8], f2_fma(W(636), adj[6], f2_mul(W(37), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(725), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_fma(W(826), adj[8], f2_fma(W(637), adj[6], f2_mul(W(38), adj[0]))); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[4], g[1]); g[4] = f2_fma(v, x[1], g[4]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); unsigned long long v; v = f2_mul(W(208), adj[2]); { const unsigned long long s = f2_mul(W(131), adj[1]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(231), adj[2]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(332), adj[3]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(232), adj[2]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(534), adj[5]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(442), adj[4]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(535), adj[5]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_fma(W(827), adj[8], f2_fma(W(638), adj[6], f2_mul(W(39), adj[0]))); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(726), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_fma(W(828), adj[8], f2_fma(W(639), adj[6], f2_mul(W(40), adj[0]))); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(727), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[5], g[1]); g[5] = f2_fma(v, x[1], g[5]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); unsigned long long v; v = f2_mul(W(96), adj[1]); { const unsigned long long s = f2_mul(W(132), adj[1]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(133), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(829), adj[8]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(728), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_fma(W(830), adj[8], f2_fma(W(640), adj[6], f2_mul(W(41), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(536), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(443), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(537), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(444), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[6], g[1]); g[6] = f2_fma(v, x[1], g[6]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(134), adj[1]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } { const unsigned long long s = f2_mul(W(729), adj[7]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_fma(W(831), adj[8], f2_fma(W(641), adj[6], f2_mul(W(42), adj[0]))); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(730), adj[7]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(445), adj[4]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(538), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(446), adj[4]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(539), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[7], g[1]); g[7] = f2_fma(v, x[1], g[7]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); unsigned long long v; v = f2_mul(W(97), adj[1]); { const unsigned long long s = f2_mul(W(135), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_fma(W(832), adj[8], f2_fma(W(642), adj[6], f2_mul(W(43), adj[0]))); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(731), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_fma(W(833), adj[8], f2_fma(W(643), adj[6], f2_mul(W(44), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(540), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(447), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(541), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(448), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[8], g[1]); g[8] = f2_fma(v, x[1], g[8]); } \
      { const unsigned long long p = f2_mul(x[1], x[9]); unsigned long long v; v = f2_mul(W(792), adj[8]); { const unsigned long long s = f2_mul(W(136), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(137), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(333), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(233), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[9], g[1]); g[9] = f2_fma(v, x[1], g[9]); } \
      { const unsigned long long p = f2_mul(x[1], x[10]); unsigned long long v; v = f2_mul(W(694), adj[7]); { const unsigned long long s = f2_mul(W(138), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(334), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(234), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(235), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[10], g[1]); g[10] = f2_fma(v, x[1], g[10]); } \
      { const unsigned long long p = f2_mul(x[1], x[11]); unsigned long long v; v = f2_fma(W(793), adj[8], f2_mul(W(600), adj[6])); { const unsigned long long s = f2_mul(W(139), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(236), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(335), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(237), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(336), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[11], g[1]); g[11] = f2_fma(v, x[1], g[11]); } \
      { const unsigned long long p = f2_mul(x[1], x[12]); unsigned long long v; v = f2_mul(W(503), adj[5]); { const unsigned long long s = f2_mul(W(140), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(141), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[12], g[1]); g[12] = f2_fma(v, x[1], g[12]); } \
      { const unsigned long long p = f2_mul(x[1], x[13]); unsigned long long v; v = f2_mul(W(413), adj[4]); { const unsigned long long s = f2_mul(W(142), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(143), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[13], g[1]); g[13] = f2_fma(v, x[1], g[13]); } \
      { const unsigned long long p = f2_mul(x[1], x[14]); unsigned long long v; v = f2_mul(W(504), adj[5]); { const unsigned long long s = f2_mul(W(144), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[14], g[1]); g[14] = f2_fma(v, x[1], g[14]); } \
      { const unsigned long long p = f2_mul(x[1], x[15]); unsigned long long v; v = f2_mul(W(414), adj[4]); { const unsigned long long s = f2_mul(W(145), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[15], g[1]); g[15] = f2_fma(v, x[1], g[15]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); unsigned long long v; v = f2_fma(W(601), adj[6], f2_mul(W(3), adj[0])); { const unsigned long long s = f2_mul(W(238), adj[2]); g[2] = f2_fma(s, p, g[2]); v = f2_fma(s, x[2], v); } { const unsigned long long s = f2_mul(W(337), adj[3]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(449), adj[4]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(542), adj[5]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_fma(W(644), adj[6], f2_mul(W(45), adj[0])); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(732), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(834), adj[8]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(146), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(239), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(338), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[2] = f2_fma(v, x[2], g[2]); g[2] = f2_fma(v, x[2], g[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); unsigned long long v; v = f2_mul(W(695), adj[7]); { const unsigned long long s = f2_mul(W(240), adj[2]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(543), adj[5]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(450), adj[4]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(733), adj[7]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_fma(W(835), adj[8], f2_fma(W(645), adj[6], f2_mul(W(46), adj[0]))); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(734), adj[7]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(147), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(339), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(241), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(340), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[3], g[2]); g[3] = f2_fma(v, x[2], g[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(242), adj[2]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } { const unsigned long long s = f2_mul(W(341), adj[3]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(148), adj[1]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(735), adj[7]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_fma(W(646), adj[6], f2_mul(W(47), adj[0])); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(736), adj[7]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(451), adj[4]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(544), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(545), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[2] = f2_fma(v, x[4], g[2]); g[4] = f2_fma(v, x[2], g[4]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); unsigned long long v; v = f2_mul(W(98), adj[1]); { const unsigned long long s = f2_mul(W(243), adj[2]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(149), adj[1]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(150), adj[1]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(836), adj[8]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(737), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_fma(W(837), adj[8], f2_fma(W(647), adj[6], f2_mul(W(48), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(546), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(452), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(547), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(453), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[2] = f2_fma(v, x[5], g[2]); g[5] = f2_fma(v, x[2], g[5]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); unsigned long long v; v = f2_mul(W(209), adj[2]); { const unsigned long long s = f2_mul(W(244), adj[2]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(342), adj[3]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(454), adj[4]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(548), adj[5]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_fma(W(648), adj[6], f2_mul(W(49), adj[0])); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(738), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(838), adj[8]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[6], g[2]); g[6] = f2_fma(v, x[2], g[6]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); unsigned long long v; v = f2_mul(W(301), adj[3]); { const unsigned long long s = f2_mul(W(245), adj[2]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(343), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(455), adj[4]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(549), adj[5]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(456), adj[4]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(739), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(839), adj[8], f2_fma(W(649), adj[6], f2_mul(W(50), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(740), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(840), adj[8]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[2] = f2_fma(v, x[7], g[2]); g[7] = f2_fma(v, x[2], g[7]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(246), adj[2]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } { const unsigned long long s = f2_mul(W(550), adj[5]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(551), adj[5]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(841), adj[8]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(741), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_fma(W(650), adj[6], f2_mul(W(51), adj[0])); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(742), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[2] = f2_fma(v, x[8], g[2]); g[8] = f2_fma(v, x[2], g[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(247), adj[2]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(344), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(151), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[9], g[2]); g[9] = f2_fma(v, x[2], g[9]); } \
      { const unsigned long long p = f2_mul(x[2], x[10]); unsigned long long v; v = f2_mul(W(415), adj[4]); { const unsigned long long s = f2_mul(W(248), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(345), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(152), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(153), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[2] = f2_fma(v, x[10], g[2]); g[10] = f2_fma(v, x[2], g[10]); } \
      { const unsigned long long p = f2_mul(x[2], x[11]); unsigned long long v; v = f2_mul(W(505), adj[5]); { const unsigned long long s = f2_mul(W(249), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(154), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(155), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[11], g[2]); g[11] = f2_fma(v, x[2], g[11]); } \
      { const unsigned long long p = f2_mul(x[2], x[12]); unsigned long long v; v = f2_mul(W(602), adj[6]); { const unsigned long long s = f2_mul(W(250), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(346), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[2] = f2_fma(v, x[12], g[2]); g[12] = f2_fma(v, x[2], g[12]); } \
      { const unsigned long long p = f2_mul(x[2], x[13]); unsigned long long v; v = f2_mul(W(696), adj[7]); { const unsigned long long s = f2_mul(W(251), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(347), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[2] = f2_fma(v, x[13], g[2]); g[13] = f2_fma(v, x[2], g[13]); } \
      { const unsigned long long p = f2_mul(x[2], x[14]); unsigned long long v; v = f2_mul(W(794), adj[8]); { const unsigned long long s = f2_mul(W(252), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(348), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[2] = f2_fma(v, x[14], g[2]); g[14] = f2_fma(v, x[2], g[14]); } \
      { const unsigned long long p = f2_mul(x[2], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(253), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[2] = f2_fma(v, x[15], g[2]); g[15] = f2_fma(v, x[2], g[15]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); unsigned long long v; v = f2_fma(W(795), adj[8], f2_fma(W(603), adj[6], f2_mul(W(4), adj[0]))); { const unsigned long long s = f2_mul(W(349), adj[3]); g[3] = f2_fma(s, p, g[3]); v = f2_fma(s, x[3], v); } { const unsigned long long s = f2_mul(W(457), adj[4]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(552), adj[5]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_fma(W(842), adj[8], f2_fma(W(651), adj[6], f2_mul(W(52), adj[0]))); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(743), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_fma(W(843), adj[8], f2_fma(W(652), adj[6], f2_mul(W(53), adj[0]))); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(156), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(157), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(254), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(350), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(255), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(351), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[3], g[3]); g[3] = f2_fma(v, x[3], g[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); unsigned long long v; v = f2_mul(W(99), adj[1]); { const unsigned long long s = f2_mul(W(352), adj[3]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(256), adj[2]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(158), adj[1]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_fma(W(844), adj[8], f2_fma(W(653), adj[6], f2_mul(W(54), adj[0]))); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(744), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_fma(W(845), adj[8], f2_fma(W(654), adj[6], f2_mul(W(55), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(553), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(458), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(554), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(459), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[4], g[3]); g[4] = f2_fma(v, x[3], g[4]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(353), adj[3]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } { const unsigned long long s = f2_mul(W(159), adj[1]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(745), adj[7]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_fma(W(846), adj[8], f2_fma(W(655), adj[6], f2_mul(W(56), adj[0]))); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(746), adj[7]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(460), adj[4]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(555), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(461), adj[4]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(556), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[5], g[3]); g[5] = f2_fma(v, x[3], g[5]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); unsigned long long v; v = f2_mul(W(302), adj[3]); { const unsigned long long s = f2_mul(W(354), adj[3]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(257), adj[2]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(355), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(462), adj[4]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(557), adj[5]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(463), adj[4]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(747), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(847), adj[8], f2_fma(W(656), adj[6], f2_mul(W(57), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(748), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(848), adj[8]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[6], g[3]); g[6] = f2_fma(v, x[3], g[6]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); unsigned long long v; v = f2_mul(W(210), adj[2]); { const unsigned long long s = f2_mul(W(356), adj[3]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(258), adj[2]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(558), adj[5]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(464), adj[4]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(559), adj[5]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_fma(W(849), adj[8], f2_fma(W(657), adj[6], f2_mul(W(58), adj[0]))); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(749), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_fma(W(850), adj[8], f2_fma(W(658), adj[6], f2_mul(W(59), adj[0]))); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(750), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[7], g[3]); g[7] = f2_fma(v, x[3], g[7]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); unsigned long long v; v = f2_mul(W(303), adj[3]); { const unsigned long long s = f2_mul(W(357), adj[3]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(465), adj[4]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(560), adj[5]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(466), adj[4]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(751), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(851), adj[8], f2_fma(W(659), adj[6], f2_mul(W(60), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(752), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_fma(W(852), adj[8], f2_fma(W(660), adj[6], f2_mul(W(61), adj[0]))); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[8], g[3]); g[8] = f2_fma(v, x[3], g[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[9]); unsigned long long v; v = f2_mul(W(416), adj[4]); { const unsigned long long s = f2_mul(W(358), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(259), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(359), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(160), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[3] = f2_fma(v, x[9], g[3]); g[9] = f2_fma(v, x[3], g[9]); } \
      { const unsigned long long p = f2_mul(x[3], x[10]); unsigned long long v; v = f2_mul(W(506), adj[5]); { const unsigned long long s = f2_mul(W(360), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(260), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(161), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } g[3] = f2_fma(v, x[10], g[3]); g[10] = f2_fma(v, x[3], g[10]); } \
      { const unsigned long long p = f2_mul(x[3], x[11]); unsigned long long v; v = f2_mul(W(417), adj[4]); { const unsigned long long s = f2_mul(W(361), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(162), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(163), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[11], g[3]); g[11] = f2_fma(v, x[3], g[11]); } \
      { const unsigned long long p = f2_mul(x[3], x[12]); unsigned long long v; v = f2_mul(W(697), adj[7]); { const unsigned long long s = f2_mul(W(362), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(261), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(363), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[3] = f2_fma(v, x[12], g[3]); g[12] = f2_fma(v, x[3], g[12]); } \
      { const unsigned long long p = f2_mul(x[3], x[13]); unsigned long long v; v = f2_fma(W(796), adj[8], f2_mul(W(604), adj[6])); { const unsigned long long s = f2_mul(W(364), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(262), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(365), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[13], g[3]); g[13] = f2_fma(v, x[3], g[13]); } \
      { const unsigned long long p = f2_mul(x[3], x[14]); unsigned long long v; v = f2_mul(W(698), adj[7]); { const unsigned long long s = f2_mul(W(366), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(263), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[14], g[3]); g[14] = f2_fma(v, x[3], g[14]); } \
      { const unsigned long long p = f2_mul(x[3], x[15]); unsigned long long v; v = f2_mul(W(797), adj[8]); { const unsigned long long s = f2_mul(W(367), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[15], g[3]); g[15] = f2_fma(v, x[3], g[15]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); unsigned long long v; v = f2_fma(W(605), adj[6], f2_mul(W(5), adj[0])); { const unsigned long long s = f2_mul(W(467), adj[4]); g[4] = f2_fma(s, p, g[4]); v = f2_fma(s, x[4], v); } { const unsigned long long s = f2_mul(W(561), adj[5]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_fma(W(661), adj[6], f2_mul(W(62), adj[0])); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(753), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(853), adj[8]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(164), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(165), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(264), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(368), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(369), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[4], g[4]); g[4] = f2_fma(v, x[4], g[4]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); unsigned long long v; v = f2_mul(W(699), adj[7]); { const unsigned long long s = f2_mul(W(468), adj[4]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_mul(W(63), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(166), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(370), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(265), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(371), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(266), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[5], g[4]); g[5] = f2_fma(v, x[4], g[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[6]); unsigned long long v; v = f2_mul(W(418), adj[4]); { const unsigned long long s = f2_mul(W(469), adj[4]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(372), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(267), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(373), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(167), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(168), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[6], g[4]); g[6] = f2_fma(v, x[4], g[6]); } \
      { const unsigned long long p = f2_mul(x[4], x[7]); unsigned long long v; v = f2_mul(W(507), adj[5]); { const unsigned long long s = f2_mul(W(470), adj[4]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(268), adj[2]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(374), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(269), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(169), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(170), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[4] = f2_fma(v, x[7], g[4]); g[7] = f2_fma(v, x[4], g[7]); } \
      { const unsigned long long p = f2_mul(x[4], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(471), adj[4]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } { const unsigned long long s = f2_mul(W(375), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(171), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[8], g[4]); g[8] = f2_fma(v, x[4], g[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); unsigned long long v; v = f2_mul(W(304), adj[3]); { const unsigned long long s = f2_mul(W(472), adj[4]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(562), adj[5]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(473), adj[4]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(754), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(854), adj[8], f2_fma(W(662), adj[6], f2_mul(W(64), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(755), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[4] = f2_fma(v, x[9], g[4]); g[9] = f2_fma(v, x[4], g[9]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); unsigned long long v; v = f2_mul(W(211), adj[2]); { const unsigned long long s = f2_mul(W(474), adj[4]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(563), adj[5]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_fma(W(663), adj[6], f2_mul(W(65), adj[0])); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(756), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(855), adj[8]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(757), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[10], g[4]); g[10] = f2_fma(v, x[4], g[10]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); unsigned long long v; v = f2_mul(W(305), adj[3]); { const unsigned long long s = f2_mul(W(475), adj[4]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(758), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(664), adj[6], f2_mul(W(66), adj[0])); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(759), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_fma(W(856), adj[8], f2_fma(W(665), adj[6], f2_mul(W(67), adj[0]))); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[11], g[4]); g[11] = f2_fma(v, x[4], g[11]); } \
      { const unsigned long long p = f2_mul(x[4], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(476), adj[4]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(564), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(565), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[12], g[4]); g[12] = f2_fma(v, x[4], g[12]); } \
      { const unsigned long long p = f2_mul(x[4], x[13]); unsigned long long v; v = f2_mul(W(100), adj[1]); { const unsigned long long s = f2_mul(W(477), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(566), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(478), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[13], g[4]); g[13] = f2_fma(v, x[4], g[13]); } \
      { const unsigned long long p = f2_mul(x[4], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(479), adj[4]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } { const unsigned long long s = f2_mul(W(567), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[14], g[4]); g[14] = f2_fma(v, x[4], g[14]); } \
      { const unsigned long long p = f2_mul(x[4], x[15]); unsigned long long v; v = f2_mul(W(101), adj[1]); { const unsigned long long s = f2_mul(W(480), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[15], g[4]); g[15] = f2_fma(v, x[4], g[15]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); unsigned long long v; v = f2_fma(W(798), adj[8], f2_fma(W(606), adj[6], f2_mul(W(6), adj[0]))); { const unsigned long long s = f2_mul(W(568), adj[5]); g[5] = f2_fma(s, p, g[5]); v = f2_fma(s, x[5], v); } { const unsigned long long s = f2_fma(W(666), adj[6], f2_mul(W(68), adj[0])); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(760), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_fma(W(857), adj[8], f2_mul(W(69), adj[0])); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(172), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(173), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(270), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(376), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(271), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(377), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[5], g[5]); g[5] = f2_fma(v, x[5], g[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[6]); unsigned long long v; v = f2_mul(W(508), adj[5]); { const unsigned long long s = f2_mul(W(569), adj[5]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(378), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(272), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(174), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(175), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[6], g[5]); g[6] = f2_fma(v, x[5], g[6]); } \
      { const unsigned long long p = f2_mul(x[5], x[7]); unsigned long long v; v = f2_mul(W(419), adj[4]); { const unsigned long long s = f2_mul(W(570), adj[5]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(379), adj[3]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(273), adj[2]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(380), adj[3]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(176), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(177), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[7], g[5]); g[7] = f2_fma(v, x[5], g[7]); } \
      { const unsigned long long p = f2_mul(x[5], x[8]); unsigned long long v; v = f2_mul(W(509), adj[5]); { const unsigned long long s = f2_mul(W(571), adj[5]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(274), adj[2]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(381), adj[3]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(275), adj[2]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(178), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(179), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[8], g[5]); g[8] = f2_fma(v, x[5], g[8]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(572), adj[5]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(481), adj[4]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(573), adj[5]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(858), adj[8]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(761), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_fma(W(859), adj[8], f2_fma(W(667), adj[6], f2_mul(W(70), adj[0]))); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[9], g[5]); g[9] = f2_fma(v, x[5], g[9]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); unsigned long long v; v = f2_mul(W(306), adj[3]); { const unsigned long long s = f2_mul(W(574), adj[5]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(482), adj[4]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(762), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(860), adj[8], f2_fma(W(668), adj[6], f2_mul(W(71), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_fma(W(861), adj[8], f2_fma(W(669), adj[6], f2_mul(W(72), adj[0]))); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[10], g[5]); g[10] = f2_fma(v, x[5], g[10]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); unsigned long long v; v = f2_mul(W(212), adj[2]); { const unsigned long long s = f2_mul(W(575), adj[5]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_fma(W(862), adj[8], f2_fma(W(670), adj[6], f2_mul(W(73), adj[0]))); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(763), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_fma(W(863), adj[8], f2_fma(W(671), adj[6], f2_mul(W(74), adj[0]))); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(764), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[11], g[5]); g[11] = f2_fma(v, x[5], g[11]); } \
      { const unsigned long long p = f2_mul(x[5], x[12]); unsigned long long v; v = f2_mul(W(102), adj[1]); { const unsigned long long s = f2_mul(W(576), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(483), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(577), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(484), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[12], g[5]); g[12] = f2_fma(v, x[5], g[12]); } \
      { const unsigned long long p = f2_mul(x[5], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(578), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(485), adj[4]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(579), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[13], g[5]); g[13] = f2_fma(v, x[5], g[13]); } \
      { const unsigned long long p = f2_mul(x[5], x[14]); unsigned long long v; v = f2_mul(W(103), adj[1]); { const unsigned long long s = f2_mul(W(580), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(486), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[14], g[5]); g[14] = f2_fma(v, x[5], g[14]); } \
      { const unsigned long long p = f2_mul(x[5], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(581), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[5] = f2_fma(v, x[15], g[5]); g[15] = f2_fma(v, x[5], g[15]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); unsigned long long v; v = f2_fma(W(607), adj[6], f2_mul(W(7), adj[0])); { const unsigned long long s = f2_fma(W(672), adj[6], f2_mul(W(75), adj[0])); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(765), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(864), adj[8]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(180), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(276), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(382), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[6] = f2_fma(v, x[6], g[6]); g[6] = f2_fma(v, x[6], g[6]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); unsigned long long v; v = f2_mul(W(700), adj[7]); { const unsigned long long s = f2_fma(W(673), adj[6], f2_mul(W(76), adj[0])); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_mul(W(181), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(383), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(277), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(384), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[6] = f2_fma(v, x[7], g[6]); g[7] = f2_fma(v, x[6], g[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); unsigned long long v; v = f2_mul(W(799), adj[8]); { const unsigned long long s = f2_fma(W(674), adj[6], f2_mul(W(77), adj[0])); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(182), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(183), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(385), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(278), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(386), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[6] = f2_fma(v, x[8], g[6]); g[8] = f2_fma(v, x[6], g[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); unsigned long long v; { const unsigned long long s = f2_fma(W(675), adj[6], f2_mul(W(78), adj[0])); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(766), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(865), adj[8]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(487), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(582), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[6] = f2_fma(v, x[9], g[6]); g[9] = f2_fma(v, x[6], g[9]); } \
      { const unsigned long long p = f2_mul(x[6], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(676), adj[6]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(767), adj[7]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(488), adj[4]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(583), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(584), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[6] = f2_fma(v, x[10], g[6]); g[10] = f2_fma(v, x[6], g[10]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); unsigned long long v; v = f2_mul(W(104), adj[1]); { const unsigned long long s = f2_fma(W(866), adj[8], f2_fma(W(677), adj[6], f2_mul(W(79), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(585), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(489), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(586), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(490), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[6] = f2_fma(v, x[11], g[6]); g[11] = f2_fma(v, x[6], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); unsigned long long v; v = f2_mul(W(213), adj[2]); { const unsigned long long s = f2_fma(W(678), adj[6], f2_mul(W(80), adj[0])); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(768), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(867), adj[8]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[6] = f2_fma(v, x[12], g[6]); g[12] = f2_fma(v, x[6], g[12]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); unsigned long long v; v = f2_mul(W(307), adj[3]); { const unsigned long long s = f2_fma(W(868), adj[8], f2_fma(W(679), adj[6], f2_mul(W(81), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(769), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(869), adj[8]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[6] = f2_fma(v, x[13], g[6]); g[13] = f2_fma(v, x[6], g[13]); } \
      { const unsigned long long p = f2_mul(x[6], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(680), adj[6]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } { const unsigned long long s = f2_mul(W(770), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[6] = f2_fma(v, x[14], g[6]); g[14] = f2_fma(v, x[6], g[14]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); unsigned long long v; { const unsigned long long s = f2_fma(W(681), adj[6], f2_mul(W(82), adj[0])); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[6] = f2_fma(v, x[15], g[6]); g[15] = f2_fma(v, x[6], g[15]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); unsigned long long v; v = f2_fma(W(800), adj[8], f2_fma(W(608), adj[6], f2_mul(W(8), adj[0]))); { const unsigned long long s = f2_mul(W(771), adj[7]); g[7] = f2_fma(s, p, g[7]); v = f2_fma(s, x[7], v); } { const unsigned long long s = f2_fma(W(870), adj[8], f2_mul(W(83), adj[0])); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(184), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(185), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(279), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(387), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(280), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(388), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[7], g[7]); g[7] = f2_fma(v, x[7], g[7]); } \
      { const unsigned long long p = f2_mul(x[7], x[8]); unsigned long long v; v = f2_mul(W(701), adj[7]); { const unsigned long long s = f2_mul(W(772), adj[7]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(186), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(389), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(281), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(390), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(282), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[8], g[7]); g[8] = f2_fma(v, x[7], g[8]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(773), adj[7]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_fma(W(871), adj[8], f2_fma(W(682), adj[6], f2_mul(W(84), adj[0]))); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(774), adj[7]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(491), adj[4]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(587), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(492), adj[4]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[7] = f2_fma(v, x[9], g[7]); g[9] = f2_fma(v, x[7], g[9]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); unsigned long long v; v = f2_mul(W(105), adj[1]); { const unsigned long long s = f2_mul(W(775), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_fma(W(872), adj[8], f2_fma(W(683), adj[6], f2_mul(W(85), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(588), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(493), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(494), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[10], g[7]); g[10] = f2_fma(v, x[7], g[10]); } \
      { const unsigned long long p = f2_mul(x[7], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(776), adj[7]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } { const unsigned long long s = f2_mul(W(495), adj[4]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(589), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(496), adj[4]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(590), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[11], g[7]); g[11] = f2_fma(v, x[7], g[11]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); unsigned long long v; v = f2_mul(W(308), adj[3]); { const unsigned long long s = f2_mul(W(777), adj[7]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_fma(W(873), adj[8], f2_fma(W(684), adj[6], f2_mul(W(86), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(778), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(874), adj[8]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[12], g[7]); g[12] = f2_fma(v, x[7], g[12]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); unsigned long long v; v = f2_mul(W(214), adj[2]); { const unsigned long long s = f2_mul(W(779), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_fma(W(875), adj[8], f2_fma(W(685), adj[6], f2_mul(W(87), adj[0]))); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(780), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[13], g[7]); g[13] = f2_fma(v, x[7], g[13]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); unsigned long long v; v = f2_mul(W(309), adj[3]); { const unsigned long long s = f2_mul(W(781), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_fma(W(876), adj[8], f2_fma(W(686), adj[6], f2_mul(W(88), adj[0]))); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[7] = f2_fma(v, x[14], g[7]); g[14] = f2_fma(v, x[7], g[14]); } \
      { const unsigned long long p = f2_mul(x[7], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(782), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[7] = f2_fma(v, x[15], g[7]); g[15] = f2_fma(v, x[7], g[15]); } \
      { const unsigned long long p = f2_mul(x[8], x[8]); unsigned long long v; v = f2_fma(W(609), adj[6], f2_mul(W(9), adj[0])); { const unsigned long long s = f2_mul(W(877), adj[8]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } { const unsigned long long s = f2_mul(W(187), adj[1]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(188), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(283), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(391), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(392), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[8], g[8]); g[8] = f2_fma(v, x[8], g[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); unsigned long long v; v = f2_mul(W(106), adj[1]); { const unsigned long long s = f2_mul(W(878), adj[8]); g[9] = f2_fma(s, p, g[9]); v = f2_fma(s, x[9], v); } { const unsigned long long s = f2_mul(W(783), adj[7]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_fma(W(879), adj[8], f2_fma(W(687), adj[6], f2_mul(W(89), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(591), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(497), adj[4]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(592), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[8] = f2_fma(v, x[9], g[8]); g[9] = f2_fma(v, x[8], g[9]); } \
      { const unsigned long long p = f2_mul(x[8], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(880), adj[8]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } { const unsigned long long s = f2_mul(W(784), adj[7]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(593), adj[5]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(498), adj[4]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(594), adj[5]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[10], g[8]); g[10] = f2_fma(v, x[8], g[10]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); unsigned long long v; v = f2_mul(W(107), adj[1]); { const unsigned long long s = f2_fma(W(881), adj[8], f2_fma(W(688), adj[6], f2_mul(W(90), adj[0]))); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(595), adj[5]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(596), adj[5]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(499), adj[4]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[11], g[8]); g[11] = f2_fma(v, x[8], g[11]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(882), adj[8]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(785), adj[7]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_fma(W(689), adj[6], f2_mul(W(91), adj[0])); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(786), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[12], g[8]); g[12] = f2_fma(v, x[8], g[12]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); unsigned long long v; v = f2_mul(W(310), adj[3]); { const unsigned long long s = f2_fma(W(883), adj[8], f2_fma(W(690), adj[6], f2_mul(W(92), adj[0]))); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(787), adj[7]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_fma(W(884), adj[8], f2_fma(W(691), adj[6], f2_mul(W(93), adj[0]))); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[13], g[8]); g[13] = f2_fma(v, x[8], g[13]); } \
      { const unsigned long long p = f2_mul(x[8], x[14]); unsigned long long v; v = f2_mul(W(215), adj[2]); { const unsigned long long s = f2_mul(W(885), adj[8]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(788), adj[7]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[14], g[8]); g[14] = f2_fma(v, x[8], g[14]); } \
      { const unsigned long long p = f2_mul(x[8], x[15]); unsigned long long v; v = f2_mul(W(311), adj[3]); { const unsigned long long s = f2_mul(W(886), adj[8]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[15], g[8]); g[15] = f2_fma(v, x[8], g[15]); } \
      { const unsigned long long p = f2_mul(x[9], x[9]); unsigned long long v; v = f2_fma(W(610), adj[6], f2_mul(W(10), adj[0])); { const unsigned long long s = f2_mul(W(189), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(284), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(393), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[9] = f2_fma(v, x[9], g[9]); g[9] = f2_fma(v, x[9], g[9]); } \
      { const unsigned long long p = f2_mul(x[9], x[10]); unsigned long long v; v = f2_mul(W(702), adj[7]); { const unsigned long long s = f2_mul(W(190), adj[1]); g[10] = f2_fma(s, p, g[10]); v = f2_fma(s, x[10], v); } { const unsigned long long s = f2_mul(W(394), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(285), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(395), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[9] = f2_fma(v, x[10], g[9]); g[10] = f2_fma(v, x[9], g[10]); } \
      { const unsigned long long p = f2_mul(x[9], x[11]); unsigned long long v; v = f2_mul(W(801), adj[8]); { const unsigned long long s = f2_mul(W(191), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(396), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(286), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[9] = f2_fma(v, x[11], g[9]); g[11] = f2_fma(v, x[9], g[11]); } \
      { const unsigned long long p = f2_mul(x[9], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(192), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[9] = f2_fma(v, x[12], g[9]); g[12] = f2_fma(v, x[9], g[12]); } \
      { const unsigned long long p = f2_mul(x[9], x[13]); unsigned long long v; v = f2_mul(W(420), adj[4]); { const unsigned long long s = f2_mul(W(193), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[9] = f2_fma(v, x[13], g[9]); g[13] = f2_fma(v, x[9], g[13]); } \
      { const unsigned long long p = f2_mul(x[9], x[14]); unsigned long long v; v = f2_mul(W(510), adj[5]); { const unsigned long long s = f2_mul(W(194), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[9] = f2_fma(v, x[14], g[9]); g[14] = f2_fma(v, x[9], g[14]); } \
      { const unsigned long long p = f2_mul(x[10], x[10]); unsigned long long v; v = f2_mul(W(11), adj[0]); { const unsigned long long s = f2_mul(W(195), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(287), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(397), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(398), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[10] = f2_fma(v, x[10], g[10]); g[10] = f2_fma(v, x[10], g[10]); } \
      { const unsigned long long p = f2_mul(x[10], x[11]); unsigned long long v; v = f2_mul(W(703), adj[7]); { const unsigned long long s = f2_mul(W(399), adj[3]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(288), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(289), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[10] = f2_fma(v, x[11], g[10]); g[11] = f2_fma(v, x[10], g[11]); } \
      { const unsigned long long p = f2_mul(x[10], x[12]); unsigned long long v; v = f2_mul(W(421), adj[4]); { const unsigned long long s = f2_mul(W(196), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(197), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[10] = f2_fma(v, x[12], g[10]); g[12] = f2_fma(v, x[10], g[12]); } \
      { unsigned long long v; v = f2_mul(W(511), adj[5]); g[10] = f2_fma(v, x[13], g[10]); g[13] = f2_fma(v, x[10], g[13]); } \
      { const unsigned long long p = f2_mul(x[10], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(198), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[10] = f2_fma(v, x[14], g[10]); g[14] = f2_fma(v, x[10], g[14]); } \
      { unsigned long long v; v = f2_mul(W(512), adj[5]); g[10] = f2_fma(v, x[15], g[10]); g[15] = f2_fma(v, x[10], g[15]); } \
      { const unsigned long long p = f2_mul(x[11], x[11]); unsigned long long v; v = f2_fma(W(802), adj[8], f2_fma(W(611), adj[6], f2_mul(W(12), adj[0]))); { const unsigned long long s = f2_mul(W(199), adj[1]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } { const unsigned long long s = f2_mul(W(290), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(400), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(291), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(401), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[11] = f2_fma(v, x[11], g[11]); g[11] = f2_fma(v, x[11], g[11]); } \
      { const unsigned long long p = f2_mul(x[11], x[12]); unsigned long long v; v = f2_mul(W(513), adj[5]); { const unsigned long long s = f2_mul(W(200), adj[1]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(201), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[11] = f2_fma(v, x[12], g[11]); g[12] = f2_fma(v, x[11], g[12]); } \
      { const unsigned long long p = f2_mul(x[11], x[13]); unsigned long long v; v = f2_mul(W(422), adj[4]); { const unsigned long long s = f2_mul(W(202), adj[1]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(203), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[11] = f2_fma(v, x[13], g[11]); g[13] = f2_fma(v, x[11], g[13]); } \
      { const unsigned long long p = f2_mul(x[11], x[14]); unsigned long long v; v = f2_mul(W(514), adj[5]); { const unsigned long long s = f2_mul(W(204), adj[1]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[11] = f2_fma(v, x[14], g[11]); g[14] = f2_fma(v, x[11], g[14]); } \
      { const unsigned long long p = f2_mul(x[11], x[15]); unsigned long long v; v = f2_mul(W(423), adj[4]); { const unsigned long long s = f2_mul(W(205), adj[1]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[11] = f2_fma(v, x[15], g[11]); g[15] = f2_fma(v, x[11], g[15]); } \
      { const unsigned long long p = f2_mul(x[12], x[12]); unsigned long long v; v = f2_fma(W(612), adj[6], f2_mul(W(13), adj[0])); { const unsigned long long s = f2_mul(W(292), adj[2]); g[12] = f2_fma(s, p, g[12]); v = f2_fma(s, x[12], v); } { const unsigned long long s = f2_mul(W(402), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } g[12] = f2_fma(v, x[12], g[12]); g[12] = f2_fma(v, x[12], g[12]); } \
      { const unsigned long long p = f2_mul(x[12], x[13]); unsigned long long v; v = f2_mul(W(704), adj[7]); { const unsigned long long s = f2_mul(W(293), adj[2]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(403), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[12] = f2_fma(v, x[13], g[12]); g[13] = f2_fma(v, x[12], g[13]); } \
      { const unsigned long long p = f2_mul(x[12], x[14]); unsigned long long v; v = f2_mul(W(803), adj[8]); { const unsigned long long s = f2_mul(W(294), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(404), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[12] = f2_fma(v, x[14], g[12]); g[14] = f2_fma(v, x[12], g[14]); } \
      { const unsigned long long p = f2_mul(x[12], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(295), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[12] = f2_fma(v, x[15], g[12]); g[15] = f2_fma(v, x[12], g[15]); } \
      { const unsigned long long p = f2_mul(x[13], x[13]); unsigned long long v; v = f2_fma(W(804), adj[8], f2_fma(W(613), adj[6], f2_mul(W(14), adj[0]))); { const unsigned long long s = f2_mul(W(405), adj[3]); g[13] = f2_fma(s, p, g[13]); v = f2_fma(s, x[13], v); } { const unsigned long long s = f2_mul(W(296), adj[2]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(406), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[13] = f2_fma(v, x[13], g[13]); g[13] = f2_fma(v, x[13], g[13]); } \
      { const unsigned long long p = f2_mul(x[13], x[14]); unsigned long long v; v = f2_mul(W(705), adj[7]); { const unsigned long long s = f2_mul(W(407), adj[3]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } { const unsigned long long s = f2_mul(W(297), adj[2]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[13] = f2_fma(v, x[14], g[13]); g[14] = f2_fma(v, x[13], g[14]); } \
      { const unsigned long long p = f2_mul(x[13], x[15]); unsigned long long v; v = f2_mul(W(805), adj[8]); { const unsigned long long s = f2_mul(W(408), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[13] = f2_fma(v, x[15], g[13]); g[15] = f2_fma(v, x[13], g[15]); } \
      { const unsigned long long p = f2_mul(x[14], x[14]); unsigned long long v; v = f2_mul(W(15), adj[0]); { const unsigned long long s = f2_mul(W(409), adj[3]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[14] = f2_fma(v, x[14], g[14]); g[14] = f2_fma(v, x[14], g[14]); } \
      { unsigned long long v; v = f2_mul(W(706), adj[7]); g[14] = f2_fma(v, x[15], g[14]); g[15] = f2_fma(v, x[14], g[15]); } \
      { unsigned long long v; v = f2_fma(W(614), adj[6], f2_mul(W(16), adj[0])); g[15] = f2_fma(v, x[15], g[15]); g[15] = f2_fma(v, x[15], g[15]); }
#define SXB_S2_M1_FORWARD_BODY \
      o[0] = f2_fma(W(0), x[0], o[0]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); o[0] = f2_fma(p, f2_fma(W(17), x[0], W(1)), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); o[0] = f2_fma(p, f2_mul(W(18), x[1]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); o[0] = f2_fma(p, f2_mul(W(19), x[2]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); o[0] = f2_fma(p, f2_mul(W(20), x[3]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); o[0] = f2_fma(p, f2_mul(W(21), x[4]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); o[0] = f2_fma(p, f2_mul(W(22), x[5]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); o[0] = f2_fma(p, f2_mul(W(23), x[6]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); o[0] = f2_fma(p, f2_mul(W(24), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); o[0] = f2_fma(p, f2_mul(W(25), x[8]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); o[0] = f2_fma(p, f2_mul(W(26), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); o[0] = f2_fma(p, f2_mul(W(27), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); o[0] = f2_fma(p, f2_mul(W(28), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); o[0] = f2_fma(p, f2_mul(W(29), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); o[0] = f2_fma(p, f2_mul(W(30), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); o[0] = f2_fma(p, f2_mul(W(31), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); o[0] = f2_fma(p, f2_mul(W(32), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); o[0] = f2_fma(p, f2_fma(W(34), x[8], f2_fma(W(33), x[6], W(2))), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); o[0] = f2_fma(p, f2_mul(W(35), x[5]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); o[0] = f2_fma(p, f2_mul(W(36), x[4]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); o[0] = f2_fma(p, f2_fma(W(38), x[15], f2_mul(W(37), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); o[0] = f2_fma(p, f2_fma(W(40), x[14], f2_mul(W(39), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); o[0] = f2_fma(p, f2_mul(W(41), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); o[0] = f2_fma(p, f2_mul(W(42), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); o[0] = f2_fma(p, f2_fma(W(44), x[11], f2_mul(W(43), x[9])), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); o[0] = f2_fma(p, f2_fma(W(45), x[6], W(3)), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); o[0] = f2_fma(p, f2_mul(W(46), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); o[0] = f2_fma(p, f2_mul(W(47), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); o[0] = f2_fma(p, f2_mul(W(48), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); o[0] = f2_fma(p, f2_mul(W(49), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); o[0] = f2_fma(p, f2_mul(W(50), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); o[0] = f2_fma(p, f2_mul(W(51), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); o[0] = f2_fma(p, f2_fma(W(53), x[8], f2_fma(W(52), x[6], W(4))), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); o[0] = f2_fma(p, f2_fma(W(55), x[11], f2_mul(W(54), x[9])), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); o[0] = f2_fma(p, f2_mul(W(56), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); o[0] = f2_fma(p, f2_mul(W(57), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); o[0] = f2_fma(p, f2_fma(W(59), x[14], f2_mul(W(58), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); o[0] = f2_fma(p, f2_fma(W(61), x[15], f2_mul(W(60), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); o[0] = f2_fma(p, f2_fma(W(62), x[6], W(5)), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); o[0] = f2_fma(p, f2_mul(W(63), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); o[0] = f2_fma(p, f2_mul(W(64), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); o[0] = f2_fma(p, f2_mul(W(65), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); o[0] = f2_fma(p, f2_fma(W(67), x[15], f2_mul(W(66), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); o[0] = f2_fma(p, f2_fma(W(69), x[8], f2_fma(W(68), x[6], W(6))), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); o[0] = f2_fma(p, f2_mul(W(70), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); o[0] = f2_fma(p, f2_fma(W(72), x[15], f2_mul(W(71), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); o[0] = f2_fma(p, f2_fma(W(74), x[14], f2_mul(W(73), x[12])), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); o[0] = f2_fma(p, f2_fma(W(75), x[6], W(7)), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); o[0] = f2_fma(p, f2_mul(W(76), x[7]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); o[0] = f2_fma(p, f2_mul(W(77), x[8]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); o[0] = f2_fma(p, f2_mul(W(78), x[9]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); o[0] = f2_fma(p, f2_mul(W(79), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); o[0] = f2_fma(p, f2_mul(W(80), x[12]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); o[0] = f2_fma(p, f2_mul(W(81), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); o[0] = f2_fma(p, f2_mul(W(82), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); o[0] = f2_fma(p, f2_fma(W(83), x[8], W(8)), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); o[0] = f2_fma(p, f2_mul(W(84), x[10]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); o[0] = f2_fma(p, f2_mul(W(85), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); o[0] = f2_fma(p, f2_mul(W(86), x[13]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); o[0] = f2_fma(p, f2_mul(W(87), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); o[0] = f2_fma(p, f2_mul(W(88), x[15]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[8]); o[0] = f2_fma(p, W(9), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); o[0] = f2_fma(p, f2_mul(W(89), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); o[0] = f2_fma(p, f2_mul(W(90), x[11]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); o[0] = f2_fma(p, f2_mul(W(91), x[14]), o[0]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); o[0] = f2_fma(p, f2_fma(W(93), x[15], f2_mul(W(92), x[13])), o[0]); } \
      { const unsigned long long p = f2_mul(x[9], x[9]); o[0] = f2_fma(p, W(10), o[0]); } \
      { const unsigned long long p = f2_mul(x[10], x[10]); o[0] = f2_fma(p, W(11), o[0]); } \
      { const unsigned long long p = f2_mul(x[11], x[11]); o[0] = f2_fma(p, W(12), o[0]); } \
      { const unsigned long long p = f2_mul(x[12], x[12]); o[0] = f2_fma(p, W(13), o[0]); } \
      { const unsigned long long p = f2_mul(x[13], x[13]); o[0] = f2_fma(p, W(14), o[0]); } \
      { const unsigned long long p = f2_mul(x[14], x[14]); o[0] = f2_fma(p, W(15), o[0]); } \
      { const unsigned long long p = f2_mul(x[15], x[15]); o[0] = f2_fma(p, W(16), o[0]); }
#define SXB_S2_M1_REVERSE_BODY \
      g[0] = f2_fma(W(0), adj[0], g[0]); \
      { const unsigned long long p = f2_mul(x[0], x[0]); unsigned long long v; v = f2_mul(W(1), adj[0]); { const unsigned long long s = f2_mul(W(17), adj[0]); g[0] = f2_fma(s, p, g[0]); v = f2_fma(s, x[0], v); } g[0] = f2_fma(v, x[0], g[0]); g[0] = f2_fma(v, x[0], g[0]); } \
      { const unsigned long long p = f2_mul(x[0], x[1]); unsigned long long v; { const unsigned long long s = f2_mul(W(18), adj[0]); g[1] = f2_fma(s, p, g[1]); v = f2_mul(s, x[1]); } g[0] = f2_fma(v, x[1], g[0]); g[1] = f2_fma(v, x[0], g[1]); } \
      { const unsigned long long p = f2_mul(x[0], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(19), adj[0]); g[2] = f2_fma(s, p, g[2]); v = f2_mul(s, x[2]); } g[0] = f2_fma(v, x[2], g[0]); g[2] = f2_fma(v, x[0], g[2]); } \
      { const unsigned long long p = f2_mul(x[0], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(20), adj[0]); g[3] = f2_fma(s, p, g[3]); v = f2_mul(s, x[3]); } g[0] = f2_fma(v, x[3], g[0]); g[3] = f2_fma(v, x[0], g[3]); } \
      { const unsigned long long p = f2_mul(x[0], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(21), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } g[0] = f2_fma(v, x[4], g[0]); g[4] = f2_fma(v, x[0], g[4]); } \
      { const unsigned long long p = f2_mul(x[0], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(22), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } g[0] = f2_fma(v, x[5], g[0]); g[5] = f2_fma(v, x[0], g[5]); } \
      { const unsigned long long p = f2_mul(x[0], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(23), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_mul(s, x[6]); } g[0] = f2_fma(v, x[6], g[0]); g[6] = f2_fma(v, x[0], g[6]); } \
      { const unsigned long long p = f2_mul(x[0], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(24), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[0] = f2_fma(v, x[7], g[0]); g[7] = f2_fma(v, x[0], g[7]); } \
      { const unsigned long long p = f2_mul(x[0], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(25), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } g[0] = f2_fma(v, x[8], g[0]); g[8] = f2_fma(v, x[0], g[8]); } \
      { const unsigned long long p = f2_mul(x[0], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(26), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[0] = f2_fma(v, x[9], g[0]); g[9] = f2_fma(v, x[0], g[9]); } \
      { const unsigned long long p = f2_mul(x[0], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(27), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[0] = f2_fma(v, x[10], g[0]); g[10] = f2_fma(v, x[0], g[10]); } \
      { const unsigned long long p = f2_mul(x[0], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(28), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[0] = f2_fma(v, x[11], g[0]); g[11] = f2_fma(v, x[0], g[11]); } \
      { const unsigned long long p = f2_mul(x[0], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(29), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[0] = f2_fma(v, x[12], g[0]); g[12] = f2_fma(v, x[0], g[12]); } \
      { const unsigned long long p = f2_mul(x[0], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(30), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[0] = f2_fma(v, x[13], g[0]); g[13] = f2_fma(v, x[0], g[13]); } \
      { const unsigned long long p = f2_mul(x[0], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(31), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[0] = f2_fma(v, x[14], g[0]); g[14] = f2_fma(v, x[0], g[14]); } \
      { const unsigned long long p = f2_mul(x[0], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(32), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[0] = f2_fma(v, x[15], g[0]); g[15] = f2_fma(v, x[0], g[15]); } \
      { const unsigned long long p = f2_mul(x[1], x[1]); unsigned long long v; v = f2_mul(W(2), adj[0]); { const unsigned long long s = f2_mul(W(33), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(34), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[1] = f2_fma(v, x[1], g[1]); g[1] = f2_fma(v, x[1], g[1]); } \
      { const unsigned long long p = f2_mul(x[1], x[2]); unsigned long long v; { const unsigned long long s = f2_mul(W(35), adj[0]); g[5] = f2_fma(s, p, g[5]); v = f2_mul(s, x[5]); } g[1] = f2_fma(v, x[2], g[1]); g[2] = f2_fma(v, x[1], g[2]); } \
      { const unsigned long long p = f2_mul(x[1], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(36), adj[0]); g[4] = f2_fma(s, p, g[4]); v = f2_mul(s, x[4]); } g[1] = f2_fma(v, x[3], g[1]); g[3] = f2_fma(v, x[1], g[3]); } \
      { const unsigned long long p = f2_mul(x[1], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(37), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(38), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[1] = f2_fma(v, x[4], g[1]); g[4] = f2_fma(v, x[1], g[4]); } \
      { const unsigned long long p = f2_mul(x[1], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(39), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(40), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[1] = f2_fma(v, x[5], g[1]); g[5] = f2_fma(v, x[1], g[5]); } \
      { const unsigned long long p = f2_mul(x[1], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(41), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[1] = f2_fma(v, x[6], g[1]); g[6] = f2_fma(v, x[1], g[6]); } \
      { const unsigned long long p = f2_mul(x[1], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(42), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[1] = f2_fma(v, x[7], g[1]); g[7] = f2_fma(v, x[1], g[7]); } \
      { const unsigned long long p = f2_mul(x[1], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(43), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(44), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[1] = f2_fma(v, x[8], g[1]); g[8] = f2_fma(v, x[1], g[8]); } \
      { const unsigned long long p = f2_mul(x[2], x[2]); unsigned long long v; v = f2_mul(W(3), adj[0]); { const unsigned long long s = f2_mul(W(45), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[2] = f2_fma(v, x[2], g[2]); g[2] = f2_fma(v, x[2], g[2]); } \
      { const unsigned long long p = f2_mul(x[2], x[3]); unsigned long long v; { const unsigned long long s = f2_mul(W(46), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[2] = f2_fma(v, x[3], g[2]); g[3] = f2_fma(v, x[2], g[3]); } \
      { const unsigned long long p = f2_mul(x[2], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(47), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[2] = f2_fma(v, x[4], g[2]); g[4] = f2_fma(v, x[2], g[4]); } \
      { const unsigned long long p = f2_mul(x[2], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(48), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[2] = f2_fma(v, x[5], g[2]); g[5] = f2_fma(v, x[2], g[5]); } \
      { const unsigned long long p = f2_mul(x[2], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(49), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[2] = f2_fma(v, x[6], g[2]); g[6] = f2_fma(v, x[2], g[6]); } \
      { const unsigned long long p = f2_mul(x[2], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(50), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[2] = f2_fma(v, x[7], g[2]); g[7] = f2_fma(v, x[2], g[7]); } \
      { const unsigned long long p = f2_mul(x[2], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(51), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[2] = f2_fma(v, x[8], g[2]); g[8] = f2_fma(v, x[2], g[8]); } \
      { const unsigned long long p = f2_mul(x[3], x[3]); unsigned long long v; v = f2_mul(W(4), adj[0]); { const unsigned long long s = f2_mul(W(52), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(53), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[3] = f2_fma(v, x[3], g[3]); g[3] = f2_fma(v, x[3], g[3]); } \
      { const unsigned long long p = f2_mul(x[3], x[4]); unsigned long long v; { const unsigned long long s = f2_mul(W(54), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } { const unsigned long long s = f2_mul(W(55), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_fma(s, x[11], v); } g[3] = f2_fma(v, x[4], g[3]); g[4] = f2_fma(v, x[3], g[4]); } \
      { const unsigned long long p = f2_mul(x[3], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(56), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[3] = f2_fma(v, x[5], g[3]); g[5] = f2_fma(v, x[3], g[5]); } \
      { const unsigned long long p = f2_mul(x[3], x[6]); unsigned long long v; { const unsigned long long s = f2_mul(W(57), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[3] = f2_fma(v, x[6], g[3]); g[6] = f2_fma(v, x[3], g[6]); } \
      { const unsigned long long p = f2_mul(x[3], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(58), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(59), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[3] = f2_fma(v, x[7], g[3]); g[7] = f2_fma(v, x[3], g[7]); } \
      { const unsigned long long p = f2_mul(x[3], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(60), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(61), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[3] = f2_fma(v, x[8], g[3]); g[8] = f2_fma(v, x[3], g[8]); } \
      { const unsigned long long p = f2_mul(x[4], x[4]); unsigned long long v; v = f2_mul(W(5), adj[0]); { const unsigned long long s = f2_mul(W(62), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[4] = f2_fma(v, x[4], g[4]); g[4] = f2_fma(v, x[4], g[4]); } \
      { const unsigned long long p = f2_mul(x[4], x[5]); unsigned long long v; { const unsigned long long s = f2_mul(W(63), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[4] = f2_fma(v, x[5], g[4]); g[5] = f2_fma(v, x[4], g[5]); } \
      { const unsigned long long p = f2_mul(x[4], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(64), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[4] = f2_fma(v, x[9], g[4]); g[9] = f2_fma(v, x[4], g[9]); } \
      { const unsigned long long p = f2_mul(x[4], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(65), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[4] = f2_fma(v, x[10], g[4]); g[10] = f2_fma(v, x[4], g[10]); } \
      { const unsigned long long p = f2_mul(x[4], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(66), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(67), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[4] = f2_fma(v, x[11], g[4]); g[11] = f2_fma(v, x[4], g[11]); } \
      { const unsigned long long p = f2_mul(x[5], x[5]); unsigned long long v; v = f2_mul(W(6), adj[0]); { const unsigned long long s = f2_mul(W(68), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } { const unsigned long long s = f2_mul(W(69), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[5] = f2_fma(v, x[5], g[5]); g[5] = f2_fma(v, x[5], g[5]); } \
      { const unsigned long long p = f2_mul(x[5], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(70), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[5] = f2_fma(v, x[9], g[5]); g[9] = f2_fma(v, x[5], g[9]); } \
      { const unsigned long long p = f2_mul(x[5], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(71), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(72), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[5] = f2_fma(v, x[10], g[5]); g[10] = f2_fma(v, x[5], g[10]); } \
      { const unsigned long long p = f2_mul(x[5], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(73), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } { const unsigned long long s = f2_mul(W(74), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_fma(s, x[14], v); } g[5] = f2_fma(v, x[11], g[5]); g[11] = f2_fma(v, x[5], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[6]); unsigned long long v; v = f2_mul(W(7), adj[0]); { const unsigned long long s = f2_mul(W(75), adj[0]); g[6] = f2_fma(s, p, g[6]); v = f2_fma(s, x[6], v); } g[6] = f2_fma(v, x[6], g[6]); g[6] = f2_fma(v, x[6], g[6]); } \
      { const unsigned long long p = f2_mul(x[6], x[7]); unsigned long long v; { const unsigned long long s = f2_mul(W(76), adj[0]); g[7] = f2_fma(s, p, g[7]); v = f2_mul(s, x[7]); } g[6] = f2_fma(v, x[7], g[6]); g[7] = f2_fma(v, x[6], g[7]); } \
      { const unsigned long long p = f2_mul(x[6], x[8]); unsigned long long v; { const unsigned long long s = f2_mul(W(77), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_mul(s, x[8]); } g[6] = f2_fma(v, x[8], g[6]); g[8] = f2_fma(v, x[6], g[8]); } \
      { const unsigned long long p = f2_mul(x[6], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(78), adj[0]); g[9] = f2_fma(s, p, g[9]); v = f2_mul(s, x[9]); } g[6] = f2_fma(v, x[9], g[6]); g[9] = f2_fma(v, x[6], g[9]); } \
      { const unsigned long long p = f2_mul(x[6], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(79), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[6] = f2_fma(v, x[11], g[6]); g[11] = f2_fma(v, x[6], g[11]); } \
      { const unsigned long long p = f2_mul(x[6], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(80), adj[0]); g[12] = f2_fma(s, p, g[12]); v = f2_mul(s, x[12]); } g[6] = f2_fma(v, x[12], g[6]); g[12] = f2_fma(v, x[6], g[12]); } \
      { const unsigned long long p = f2_mul(x[6], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(81), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[6] = f2_fma(v, x[13], g[6]); g[13] = f2_fma(v, x[6], g[13]); } \
      { const unsigned long long p = f2_mul(x[6], x[15]); unsigned long long v; { const unsigned long long s = f2_mul(W(82), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[6] = f2_fma(v, x[15], g[6]); g[15] = f2_fma(v, x[6], g[15]); } \
      { const unsigned long long p = f2_mul(x[7], x[7]); unsigned long long v; v = f2_mul(W(8), adj[0]); { const unsigned long long s = f2_mul(W(83), adj[0]); g[8] = f2_fma(s, p, g[8]); v = f2_fma(s, x[8], v); } g[7] = f2_fma(v, x[7], g[7]); g[7] = f2_fma(v, x[7], g[7]); } \
      { const unsigned long long p = f2_mul(x[7], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(84), adj[0]); g[10] = f2_fma(s, p, g[10]); v = f2_mul(s, x[10]); } g[7] = f2_fma(v, x[9], g[7]); g[9] = f2_fma(v, x[7], g[9]); } \
      { const unsigned long long p = f2_mul(x[7], x[10]); unsigned long long v; { const unsigned long long s = f2_mul(W(85), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[7] = f2_fma(v, x[10], g[7]); g[10] = f2_fma(v, x[7], g[10]); } \
      { const unsigned long long p = f2_mul(x[7], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(86), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } g[7] = f2_fma(v, x[12], g[7]); g[12] = f2_fma(v, x[7], g[12]); } \
      { const unsigned long long p = f2_mul(x[7], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(87), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[7] = f2_fma(v, x[13], g[7]); g[13] = f2_fma(v, x[7], g[13]); } \
      { const unsigned long long p = f2_mul(x[7], x[14]); unsigned long long v; { const unsigned long long s = f2_mul(W(88), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_mul(s, x[15]); } g[7] = f2_fma(v, x[14], g[7]); g[14] = f2_fma(v, x[7], g[14]); } \
      { unsigned long long v; v = f2_mul(W(9), adj[0]); g[8] = f2_fma(v, x[8], g[8]); g[8] = f2_fma(v, x[8], g[8]); } \
      { const unsigned long long p = f2_mul(x[8], x[9]); unsigned long long v; { const unsigned long long s = f2_mul(W(89), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[8] = f2_fma(v, x[9], g[8]); g[9] = f2_fma(v, x[8], g[9]); } \
      { const unsigned long long p = f2_mul(x[8], x[11]); unsigned long long v; { const unsigned long long s = f2_mul(W(90), adj[0]); g[11] = f2_fma(s, p, g[11]); v = f2_mul(s, x[11]); } g[8] = f2_fma(v, x[11], g[8]); g[11] = f2_fma(v, x[8], g[11]); } \
      { const unsigned long long p = f2_mul(x[8], x[12]); unsigned long long v; { const unsigned long long s = f2_mul(W(91), adj[0]); g[14] = f2_fma(s, p, g[14]); v = f2_mul(s, x[14]); } g[8] = f2_fma(v, x[12], g[8]); g[12] = f2_fma(v, x[8], g[12]); } \
      { const unsigned long long p = f2_mul(x[8], x[13]); unsigned long long v; { const unsigned long long s = f2_mul(W(92), adj[0]); g[13] = f2_fma(s, p, g[13]); v = f2_mul(s, x[13]); } { const unsigned long long s = f2_mul(W(93), adj[0]); g[15] = f2_fma(s, p, g[15]); v = f2_fma(s, x[15], v); } g[8] = f2_fma(v, x[13], g[8]); g[13] = f2_fma(v, x[8], g[13]); } \
      { unsigned long long v; v = f2_mul(W(10), adj[0]); g[9] = f2_fma(v, x[9], g[9]); g[9] = f2_fma(v, x[9], g[9]); } \
      { unsigned long long v; v = f2_mul(W(11), adj[0]); g[10] = f2_fma(v, x[10], g[10]); g[10] = f2_fma(v, x[10], g[10]); } \
      { unsigned long long v; v = f2_mul(W(12), adj[0]); g[11] = f2_fma(v, x[11], g[11]); g[11] = f2_fma(v, x[11], g[11]); } \
      { unsigned long long v; v = f2_mul(W(13), adj[0]); g[12] = f2_fma(v, x[12], g[12]); g[12] = f2_fma(v, x[12], g[12]); } \
      { unsigned long long v; v = f2_mul(W(14), adj[0]); g[13] = f2_fma(v, x[13], g[13]); g[13] = f2_fma(v, x[13], g[13]); } \
      { unsigned long long v; v = f2_mul(W(15), adj[0]); g[14] = f2_fma(v, x[14], g[14]); g[14] = f2_fma(v, x[14], g[14]); } \
      { unsigned long long v; v = f2_mul(W(16), adj[0]); g[15] = f2_fma(v, x[15], g[15]); g[15] = f2_fma(v, x[15], g[15]); }
#define SXB_S2_ROW_BATCHES 24
#define SXB_S2_L1_REVERSE_EDGE_BODY \
    { f2 y[1]; load_pair_harmonics<0>(yrow, y); \
    { /* path 0: edge l=0, source l=0 -> l=0 */ RADIAL(0) f2 yw, t[1], v[1]; \
      t[0] = f2_mul(R, y[0]); \
      ROWS(0) { const f2 w = rows[0]; v[0] = f2_mul(h[0], w); hadj[0] = f2_mul(t[0], w); } \
      yw = f2_mul(y[0], v[0]); \
      radial = f2_mul(dR, yw); \
    } \
    { /* path 4: edge l=0, source l=1 -> l=1 */ RADIAL(4) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[1]; v[0] = f2_mul(h[1], w); hadj[1] = f2_mul(t[0], w); } \
      { const f2 w = rows[2]; v[0] = f2_fma(h[2], w, v[0]); hadj[2] = f2_mul(t[0], w); } \
      { const f2 w = rows[3]; v[0] = f2_fma(h[3], w, v[0]); hadj[3] = f2_mul(t[0], w); } \
      yw = f2_mul(y[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 11: edge l=0, source l=2 -> l=2 */ RADIAL(11) f2 yw, t[5], v[5]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[4]; v[0] = f2_mul(h[4], w); hadj[4] = f2_mul(t[0], w); } \
      { const f2 w = rows[5]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_mul(t[0], w); } \
      { const f2 w = rows[6]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_mul(t[0], w); } \
      { const f2 w = rows[7]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_mul(t[0], w); } \
      ROWS(1) { const f2 w = rows[0]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_mul(t[0], w); } \
      yw = f2_mul(y[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
    } \
    { f2 y[3], ang[3]; load_pair_harmonics<1>(yrow, y); \
    { /* path 1: edge l=1, source l=1 -> l=0 */ RADIAL(1) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[1]; v[0] = f2_mul(h[1], w); hadj[1] = f2_fma(t[0], w, hadj[1]); } \
      ang[0] = f2_mul(R, v[0]); yw = f2_mul(y[0], v[0]); \
      t[0] = f2_mul(R, y[1]); \
      { const f2 w = rows[2]; v[0] = f2_mul(h[2], w); hadj[2] = f2_fma(t[0], w, hadj[2]); } \
      ang[1] = f2_mul(R, v[0]); yw = f2_fma(y[1], v[0], yw); \
      t[0] = f2_mul(R, y[2]); \
      { const f2 w = rows[3]; v[0] = f2_mul(h[3], w); hadj[3] = f2_fma(t[0], w, hadj[3]); } \
      ang[2] = f2_mul(R, v[0]); yw = f2_fma(y[2], v[0], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 3: edge l=1, source l=0 -> l=1 */ RADIAL(3) f2 yw, t[1], v[1]; \
      t[0] = f2_mul(R, h[0]); \
      { const f2 w = rows[4]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[5]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[6]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      hadj[0] = f2_fma(R, v[0], hadj[0]); yw = f2_mul(h[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 6: edge l=1, source l=2 -> l=1 */ RADIAL(6) f2 yw, t[5], v[5]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[7]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      ROWS(2) { const f2 w = rows[0]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      { const f2 w = rows[2]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[0] = f2_fma(R, v[0], ang[0]); yw = f2_mul(y[0], v[0]); \
      t[0] = f2_mul(R, y[1]); \
      { const f2 w = rows[3]; v[0] = f2_mul(h[5], w); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[4]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      { const f2 w = rows[5]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      ang[1] = f2_fma(R, v[0], ang[1]); yw = f2_fma(y[1], v[0], yw); \
      t[0] = f2_mul(R, y[2]); \
      { const f2 w = rows[6]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      { const f2 w = rows[7]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      ROWS(3) { const f2 w = rows[0]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[2] = f2_fma(R, v[0], ang[2]); yw = f2_fma(y[2], v[0], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 9: edge l=1, source l=1 -> l=2 */ RADIAL(9) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[2]; v[0] = f2_mul(h[1], w); hadj[1] = f2_fma(t[0], w, hadj[1]); } \
      { const f2 w = rows[3]; v[0] = f2_fma(h[2], w, v[0]); hadj[2] = f2_fma(t[0], w, hadj[2]); } \
      { const f2 w = rows[4]; v[0] = f2_fma(h[3], w, v[0]); hadj[3] = f2_fma(t[0], w, hadj[3]); } \
      ang[0] = f2_fma(R, v[0], ang[0]); yw = f2_mul(y[0], v[0]); \
      t[0] = f2_mul(R, y[1]); \
      { const f2 w = rows[5]; v[0] = f2_mul(h[1], w); hadj[1] = f2_fma(t[0], w, hadj[1]); } \
      { const f2 w = rows[6]; v[0] = f2_fma(h[2], w, v[0]); hadj[2] = f2_fma(t[0], w, hadj[2]); } \
      { const f2 w = rows[7]; v[0] = f2_fma(h[3], w, v[0]); hadj[3] = f2_fma(t[0], w, hadj[3]); } \
      ang[1] = f2_fma(R, v[0], ang[1]); yw = f2_fma(y[1], v[0], yw); \
      t[0] = f2_mul(R, y[2]); \
      ROWS(4) { const f2 w = rows[0]; v[0] = f2_mul(h[1], w); hadj[1] = f2_fma(t[0], w, hadj[1]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[2], w, v[0]); hadj[2] = f2_fma(t[0], w, hadj[2]); } \
      { const f2 w = rows[2]; v[0] = f2_fma(h[3], w, v[0]); hadj[3] = f2_fma(t[0], w, hadj[3]); } \
      ang[2] = f2_fma(R, v[0], ang[2]); yw = f2_fma(y[2], v[0], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 15: edge l=1, source l=2 -> l=3 */ RADIAL(15) f2 yw, t[5], v[5]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[3]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      { const f2 w = rows[4]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[5]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      { const f2 w = rows[6]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      { const f2 w = rows[7]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[0] = f2_fma(R, v[0], ang[0]); yw = f2_mul(y[0], v[0]); \
      t[0] = f2_mul(R, y[1]); \
      ROWS(5) { const f2 w = rows[0]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[2]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      { const f2 w = rows[3]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      { const f2 w = rows[4]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[1] = f2_fma(R, v[0], ang[1]); yw = f2_fma(y[1], v[0], yw); \
      t[0] = f2_mul(R, y[2]); \
      { const f2 w = rows[5]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      { const f2 w = rows[6]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[7]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      ROWS(6) { const f2 w = rows[0]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[2] = f2_fma(R, v[0], ang[2]); yw = f2_fma(y[2], v[0], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
      f[1] = f2_sum(ang[0]); f[2] = f2_sum(ang[1]); f[3] = f2_sum(ang[2]); \
    } \
    { f2 y[5], ang[5]; load_pair_harmonics<2>(yrow, y); \
    { /* path 2: edge l=2, source l=2 -> l=0 */ RADIAL(2) f2 yw, t[5], v[5]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[2]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      ang[0] = f2_mul(R, v[0]); yw = f2_mul(y[0], v[0]); \
      t[0] = f2_mul(R, y[1]); \
      { const f2 w = rows[3]; v[0] = f2_mul(h[5], w); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      ang[1] = f2_mul(R, v[0]); yw = f2_fma(y[1], v[0], yw); \
      t[0] = f2_mul(R, y[2]); \
      { const f2 w = rows[4]; v[0] = f2_mul(h[6], w); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      ang[2] = f2_mul(R, v[0]); yw = f2_fma(y[2], v[0], yw); \
      t[0] = f2_mul(R, y[3]); \
      { const f2 w = rows[5]; v[0] = f2_mul(h[7], w); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      ang[3] = f2_mul(R, v[0]); yw = f2_fma(y[3], v[0], yw); \
      t[0] = f2_mul(R, y[4]); \
      { const f2 w = rows[6]; v[0] = f2_mul(h[8], w); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[4] = f2_mul(R, v[0]); yw = f2_fma(y[4], v[0], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 5: edge l=2, source l=1 -> l=1 */ RADIAL(5) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, h[1]); \
      t[1] = f2_mul(R, h[2]); \
      t[2] = f2_mul(R, h[3]); \
      { const f2 w = rows[7]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      ROWS(7) { const f2 w = rows[0]; ang[0] = f2_fma(t[2], w, ang[0]); v[2] = f2_mul(y[0], w); } \
      { const f2 w = rows[1]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[2]; ang[1] = f2_fma(t[1], w, ang[1]); v[1] = f2_mul(y[1], w); } \
      { const f2 w = rows[3]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      { const f2 w = rows[4]; ang[2] = f2_fma(t[1], w, ang[2]); v[1] = f2_fma(y[2], w, v[1]); } \
      { const f2 w = rows[5]; ang[2] = f2_fma(t[2], w, ang[2]); v[2] = f2_fma(y[2], w, v[2]); } \
      { const f2 w = rows[6]; ang[3] = f2_fma(t[1], w, ang[3]); v[1] = f2_fma(y[3], w, v[1]); } \
      { const f2 w = rows[7]; ang[3] = f2_fma(t[2], w, ang[3]); v[2] = f2_fma(y[3], w, v[2]); } \
      ROWS(8) { const f2 w = rows[0]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[1]; ang[4] = f2_fma(t[2], w, ang[4]); v[2] = f2_fma(y[4], w, v[2]); } \
      hadj[1] = f2_fma(R, v[0], hadj[1]); yw = f2_mul(h[1], v[0]); \
      hadj[2] = f2_fma(R, v[1], hadj[2]); yw = f2_fma(h[2], v[1], yw); \
      hadj[3] = f2_fma(R, v[2], hadj[3]); yw = f2_fma(h[3], v[2], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 8: edge l=2, source l=0 -> l=2 */ RADIAL(8) f2 yw, t[1], v[1]; \
      t[0] = f2_mul(R, h[0]); \
      { const f2 w = rows[2]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[3]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[4]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      { const f2 w = rows[5]; ang[3] = f2_fma(t[0], w, ang[3]); v[0] = f2_fma(y[3], w, v[0]); } \
      { const f2 w = rows[6]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      hadj[0] = f2_fma(R, v[0], hadj[0]); yw = f2_mul(h[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 12: edge l=2, source l=2 -> l=2 */ RADIAL(12) f2 yw, t[5], v[5]; \
      t[0] = f2_mul(R, y[0]); \
      { const f2 w = rows[7]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      ROWS(9) { const f2 w = rows[0]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      { const f2 w = rows[2]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      ang[0] = f2_fma(R, v[0], ang[0]); yw = f2_mul(y[0], v[0]); \
      t[0] = f2_mul(R, y[1]); \
      { const f2 w = rows[3]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      { const f2 w = rows[4]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[5]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      { const f2 w = rows[6]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      { const f2 w = rows[7]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[1] = f2_fma(R, v[0], ang[1]); yw = f2_fma(y[1], v[0], yw); \
      t[0] = f2_mul(R, y[2]); \
      ROWS(10) { const f2 w = rows[0]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[2]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      { const f2 w = rows[3]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      { const f2 w = rows[4]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[2] = f2_fma(R, v[0], ang[2]); yw = f2_fma(y[2], v[0], yw); \
      t[0] = f2_mul(R, y[3]); \
      { const f2 w = rows[5]; v[0] = f2_mul(h[4], w); hadj[4] = f2_fma(t[0], w, hadj[4]); } \
      { const f2 w = rows[6]; v[0] = f2_fma(h[5], w, v[0]); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[7]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      ROWS(11) { const f2 w = rows[0]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      { const f2 w = rows[1]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[3] = f2_fma(R, v[0], ang[3]); yw = f2_fma(y[3], v[0], yw); \
      t[0] = f2_mul(R, y[4]); \
      { const f2 w = rows[2]; v[0] = f2_mul(h[5], w); hadj[5] = f2_fma(t[0], w, hadj[5]); } \
      { const f2 w = rows[3]; v[0] = f2_fma(h[6], w, v[0]); hadj[6] = f2_fma(t[0], w, hadj[6]); } \
      { const f2 w = rows[4]; v[0] = f2_fma(h[7], w, v[0]); hadj[7] = f2_fma(t[0], w, hadj[7]); } \
      { const f2 w = rows[5]; v[0] = f2_fma(h[8], w, v[0]); hadj[8] = f2_fma(t[0], w, hadj[8]); } \
      ang[4] = f2_fma(R, v[0], ang[4]); yw = f2_fma(y[4], v[0], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 14: edge l=2, source l=1 -> l=3 */ RADIAL(14) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, h[1]); \
      t[1] = f2_mul(R, h[2]); \
      t[2] = f2_mul(R, h[3]); \
      { const f2 w = rows[6]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[7]; ang[0] = f2_fma(t[1], w, ang[0]); v[1] = f2_mul(y[0], w); } \
      ROWS(12) { const f2 w = rows[0]; ang[0] = f2_fma(t[2], w, ang[0]); v[2] = f2_mul(y[0], w); } \
      { const f2 w = rows[1]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[2]; ang[1] = f2_fma(t[1], w, ang[1]); v[1] = f2_fma(y[1], w, v[1]); } \
      { const f2 w = rows[3]; ang[1] = f2_fma(t[2], w, ang[1]); v[2] = f2_fma(y[1], w, v[2]); } \
      { const f2 w = rows[4]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      { const f2 w = rows[5]; ang[2] = f2_fma(t[1], w, ang[2]); v[1] = f2_fma(y[2], w, v[1]); } \
      { const f2 w = rows[6]; ang[2] = f2_fma(t[2], w, ang[2]); v[2] = f2_fma(y[2], w, v[2]); } \
      { const f2 w = rows[7]; ang[3] = f2_fma(t[0], w, ang[3]); v[0] = f2_fma(y[3], w, v[0]); } \
      ROWS(13) { const f2 w = rows[0]; ang[3] = f2_fma(t[1], w, ang[3]); v[1] = f2_fma(y[3], w, v[1]); } \
      { const f2 w = rows[1]; ang[3] = f2_fma(t[2], w, ang[3]); v[2] = f2_fma(y[3], w, v[2]); } \
      { const f2 w = rows[2]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[3]; ang[4] = f2_fma(t[1], w, ang[4]); v[1] = f2_fma(y[4], w, v[1]); } \
      { const f2 w = rows[4]; ang[4] = f2_fma(t[2], w, ang[4]); v[2] = f2_fma(y[4], w, v[2]); } \
      hadj[1] = f2_fma(R, v[0], hadj[1]); yw = f2_mul(h[1], v[0]); \
      hadj[2] = f2_fma(R, v[1], hadj[2]); yw = f2_fma(h[2], v[1], yw); \
      hadj[3] = f2_fma(R, v[2], hadj[3]); yw = f2_fma(h[3], v[2], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
      f[4] = f2_sum(ang[0]); f[5] = f2_sum(ang[1]); f[6] = f2_sum(ang[2]); f[7] = f2_sum(ang[3]); f[8] = f2_sum(ang[4]); \
    } \
    { f2 y[7], ang[7]; load_pair_harmonics<3>(yrow, y); \
    { /* path 7: edge l=3, source l=2 -> l=1 */ RADIAL(7) f2 yw, t[5], v[5]; \
      t[0] = f2_mul(R, h[4]); \
      t[1] = f2_mul(R, h[5]); \
      t[2] = f2_mul(R, h[6]); \
      t[3] = f2_mul(R, h[7]); \
      t[4] = f2_mul(R, h[8]); \
      { const f2 w = rows[5]; ang[0] = f2_mul(t[0], w); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[6]; ang[0] = f2_fma(t[4], w, ang[0]); v[4] = f2_mul(y[0], w); } \
      { const f2 w = rows[7]; ang[1] = f2_mul(t[0], w); v[0] = f2_fma(y[1], w, v[0]); } \
      ROWS(14) { const f2 w = rows[0]; ang[1] = f2_fma(t[1], w, ang[1]); v[1] = f2_mul(y[1], w); } \
      { const f2 w = rows[1]; ang[1] = f2_fma(t[3], w, ang[1]); v[3] = f2_mul(y[1], w); } \
      { const f2 w = rows[2]; ang[2] = f2_mul(t[0], w); v[0] = f2_fma(y[2], w, v[0]); } \
      { const f2 w = rows[3]; ang[2] = f2_fma(t[1], w, ang[2]); v[1] = f2_fma(y[2], w, v[1]); } \
      { const f2 w = rows[4]; ang[2] = f2_fma(t[2], w, ang[2]); v[2] = f2_mul(y[2], w); } \
      { const f2 w = rows[5]; ang[2] = f2_fma(t[4], w, ang[2]); v[4] = f2_fma(y[2], w, v[4]); } \
      { const f2 w = rows[6]; ang[3] = f2_mul(t[1], w); v[1] = f2_fma(y[3], w, v[1]); } \
      { const f2 w = rows[7]; ang[3] = f2_fma(t[2], w, ang[3]); v[2] = f2_fma(y[3], w, v[2]); } \
      ROWS(15) { const f2 w = rows[0]; ang[3] = f2_fma(t[3], w, ang[3]); v[3] = f2_fma(y[3], w, v[3]); } \
      { const f2 w = rows[1]; ang[4] = f2_mul(t[0], w); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[2]; ang[4] = f2_fma(t[2], w, ang[4]); v[2] = f2_fma(y[4], w, v[2]); } \
      { const f2 w = rows[3]; ang[4] = f2_fma(t[3], w, ang[4]); v[3] = f2_fma(y[4], w, v[3]); } \
      { const f2 w = rows[4]; ang[4] = f2_fma(t[4], w, ang[4]); v[4] = f2_fma(y[4], w, v[4]); } \
      { const f2 w = rows[5]; ang[5] = f2_mul(t[1], w); v[1] = f2_fma(y[5], w, v[1]); } \
      { const f2 w = rows[6]; ang[5] = f2_fma(t[3], w, ang[5]); v[3] = f2_fma(y[5], w, v[3]); } \
      { const f2 w = rows[7]; ang[5] = f2_fma(t[4], w, ang[5]); v[4] = f2_fma(y[5], w, v[4]); } \
      ROWS(16) { const f2 w = rows[0]; ang[6] = f2_mul(t[0], w); v[0] = f2_fma(y[6], w, v[0]); } \
      { const f2 w = rows[1]; ang[6] = f2_fma(t[4], w, ang[6]); v[4] = f2_fma(y[6], w, v[4]); } \
      hadj[4] = f2_fma(R, v[0], hadj[4]); yw = f2_mul(h[4], v[0]); \
      hadj[5] = f2_fma(R, v[1], hadj[5]); yw = f2_fma(h[5], v[1], yw); \
      hadj[6] = f2_fma(R, v[2], hadj[6]); yw = f2_fma(h[6], v[2], yw); \
      hadj[7] = f2_fma(R, v[3], hadj[7]); yw = f2_fma(h[7], v[3], yw); \
      hadj[8] = f2_fma(R, v[4], hadj[8]); yw = f2_fma(h[8], v[4], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 10: edge l=3, source l=1 -> l=2 */ RADIAL(10) f2 yw, t[3], v[3]; \
      t[0] = f2_mul(R, h[1]); \
      t[1] = f2_mul(R, h[2]); \
      t[2] = f2_mul(R, h[3]); \
      { const f2 w = rows[2]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[3]; ang[0] = f2_fma(t[2], w, ang[0]); v[2] = f2_mul(y[0], w); } \
      { const f2 w = rows[4]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[5]; ang[1] = f2_fma(t[1], w, ang[1]); v[1] = f2_mul(y[1], w); } \
      { const f2 w = rows[6]; ang[1] = f2_fma(t[2], w, ang[1]); v[2] = f2_fma(y[1], w, v[2]); } \
      { const f2 w = rows[7]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      ROWS(17) { const f2 w = rows[0]; ang[2] = f2_fma(t[1], w, ang[2]); v[1] = f2_fma(y[2], w, v[1]); } \
      { const f2 w = rows[1]; ang[2] = f2_fma(t[2], w, ang[2]); v[2] = f2_fma(y[2], w, v[2]); } \
      { const f2 w = rows[2]; ang[3] = f2_fma(t[0], w, ang[3]); v[0] = f2_fma(y[3], w, v[0]); } \
      { const f2 w = rows[3]; ang[3] = f2_fma(t[1], w, ang[3]); v[1] = f2_fma(y[3], w, v[1]); } \
      { const f2 w = rows[4]; ang[3] = f2_fma(t[2], w, ang[3]); v[2] = f2_fma(y[3], w, v[2]); } \
      { const f2 w = rows[5]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[6]; ang[4] = f2_fma(t[1], w, ang[4]); v[1] = f2_fma(y[4], w, v[1]); } \
      { const f2 w = rows[7]; ang[4] = f2_fma(t[2], w, ang[4]); v[2] = f2_fma(y[4], w, v[2]); } \
      ROWS(18) { const f2 w = rows[0]; ang[5] = f2_fma(t[0], w, ang[5]); v[0] = f2_fma(y[5], w, v[0]); } \
      { const f2 w = rows[1]; ang[5] = f2_fma(t[1], w, ang[5]); v[1] = f2_fma(y[5], w, v[1]); } \
      { const f2 w = rows[2]; ang[5] = f2_fma(t[2], w, ang[5]); v[2] = f2_fma(y[5], w, v[2]); } \
      { const f2 w = rows[3]; ang[6] = f2_fma(t[0], w, ang[6]); v[0] = f2_fma(y[6], w, v[0]); } \
      { const f2 w = rows[4]; ang[6] = f2_fma(t[2], w, ang[6]); v[2] = f2_fma(y[6], w, v[2]); } \
      hadj[1] = f2_fma(R, v[0], hadj[1]); yw = f2_mul(h[1], v[0]); \
      hadj[2] = f2_fma(R, v[1], hadj[2]); yw = f2_fma(h[2], v[1], yw); \
      hadj[3] = f2_fma(R, v[2], hadj[3]); yw = f2_fma(h[3], v[2], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 13: edge l=3, source l=0 -> l=3 */ RADIAL(13) f2 yw, t[1], v[1]; \
      t[0] = f2_mul(R, h[0]); \
      { const f2 w = rows[5]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[6]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[7]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      ROWS(19) { const f2 w = rows[0]; ang[3] = f2_fma(t[0], w, ang[3]); v[0] = f2_fma(y[3], w, v[0]); } \
      { const f2 w = rows[1]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[2]; ang[5] = f2_fma(t[0], w, ang[5]); v[0] = f2_fma(y[5], w, v[0]); } \
      { const f2 w = rows[3]; ang[6] = f2_fma(t[0], w, ang[6]); v[0] = f2_fma(y[6], w, v[0]); } \
      hadj[0] = f2_fma(R, v[0], hadj[0]); yw = f2_mul(h[0], v[0]); \
      radial = f2_fma(dR, yw, radial); \
    } \
    { /* path 16: edge l=3, source l=2 -> l=3 */ RADIAL(16) f2 yw, t[5], v[5]; \
      t[0] = f2_mul(R, h[4]); \
      t[1] = f2_mul(R, h[5]); \
      t[2] = f2_mul(R, h[6]); \
      t[3] = f2_mul(R, h[7]); \
      t[4] = f2_mul(R, h[8]); \
      { const f2 w = rows[4]; ang[0] = f2_fma(t[0], w, ang[0]); v[0] = f2_mul(y[0], w); } \
      { const f2 w = rows[5]; ang[0] = f2_fma(t[1], w, ang[0]); v[1] = f2_mul(y[0], w); } \
      { const f2 w = rows[6]; ang[0] = f2_fma(t[2], w, ang[0]); v[2] = f2_mul(y[0], w); } \
      { const f2 w = rows[7]; ang[0] = f2_fma(t[3], w, ang[0]); v[3] = f2_mul(y[0], w); } \
      ROWS(20) { const f2 w = rows[0]; ang[0] = f2_fma(t[4], w, ang[0]); v[4] = f2_mul(y[0], w); } \
      { const f2 w = rows[1]; ang[1] = f2_fma(t[0], w, ang[1]); v[0] = f2_fma(y[1], w, v[0]); } \
      { const f2 w = rows[2]; ang[1] = f2_fma(t[1], w, ang[1]); v[1] = f2_fma(y[1], w, v[1]); } \
      { const f2 w = rows[3]; ang[1] = f2_fma(t[3], w, ang[1]); v[3] = f2_fma(y[1], w, v[3]); } \
      { const f2 w = rows[4]; ang[2] = f2_fma(t[0], w, ang[2]); v[0] = f2_fma(y[2], w, v[0]); } \
      { const f2 w = rows[5]; ang[2] = f2_fma(t[1], w, ang[2]); v[1] = f2_fma(y[2], w, v[1]); } \
      { const f2 w = rows[6]; ang[2] = f2_fma(t[2], w, ang[2]); v[2] = f2_fma(y[2], w, v[2]); } \
      { const f2 w = rows[7]; ang[2] = f2_fma(t[3], w, ang[2]); v[3] = f2_fma(y[2], w, v[3]); } \
      ROWS(21) { const f2 w = rows[0]; ang[2] = f2_fma(t[4], w, ang[2]); v[4] = f2_fma(y[2], w, v[4]); } \
      { const f2 w = rows[1]; ang[3] = f2_fma(t[0], w, ang[3]); v[0] = f2_fma(y[3], w, v[0]); } \
      { const f2 w = rows[2]; ang[3] = f2_fma(t[1], w, ang[3]); v[1] = f2_fma(y[3], w, v[1]); } \
      { const f2 w = rows[3]; ang[3] = f2_fma(t[2], w, ang[3]); v[2] = f2_fma(y[3], w, v[2]); } \
      { const f2 w = rows[4]; ang[3] = f2_fma(t[3], w, ang[3]); v[3] = f2_fma(y[3], w, v[3]); } \
      { const f2 w = rows[5]; ang[3] = f2_fma(t[4], w, ang[3]); v[4] = f2_fma(y[3], w, v[4]); } \
      { const f2 w = rows[6]; ang[4] = f2_fma(t[0], w, ang[4]); v[0] = f2_fma(y[4], w, v[0]); } \
      { const f2 w = rows[7]; ang[4] = f2_fma(t[1], w, ang[4]); v[1] = f2_fma(y[4], w, v[1]); } \
      ROWS(22) { const f2 w = rows[0]; ang[4] = f2_fma(t[2], w, ang[4]); v[2] = f2_fma(y[4], w, v[2]); } \
      { const f2 w = rows[1]; ang[4] = f2_fma(t[3], w, ang[4]); v[3] = f2_fma(y[4], w, v[3]); } \
      { const f2 w = rows[2]; ang[4] = f2_fma(t[4], w, ang[4]); v[4] = f2_fma(y[4], w, v[4]); } \
      { const f2 w = rows[3]; ang[5] = f2_fma(t[1], w, ang[5]); v[1] = f2_fma(y[5], w, v[1]); } \
      { const f2 w = rows[4]; ang[5] = f2_fma(t[3], w, ang[5]); v[3] = f2_fma(y[5], w, v[3]); } \
      { const f2 w = rows[5]; ang[5] = f2_fma(t[4], w, ang[5]); v[4] = f2_fma(y[5], w, v[4]); } \
      { const f2 w = rows[6]; ang[6] = f2_fma(t[0], w, ang[6]); v[0] = f2_fma(y[6], w, v[0]); } \
      { const f2 w = rows[7]; ang[6] = f2_fma(t[1], w, ang[6]); v[1] = f2_fma(y[6], w, v[1]); } \
      ROWS(23) { const f2 w = rows[0]; ang[6] = f2_fma(t[2], w, ang[6]); v[2] = f2_fma(y[6], w, v[2]); } \
      { const f2 w = rows[1]; ang[6] = f2_fma(t[3], w, ang[6]); v[3] = f2_fma(y[6], w, v[3]); } \
      { const f2 w = rows[2]; ang[6] = f2_fma(t[4], w, ang[6]); v[4] = f2_fma(y[6], w, v[4]); } \
      hadj[4] = f2_fma(R, v[0], hadj[4]); yw = f2_mul(h[4], v[0]); \
      hadj[5] = f2_fma(R, v[1], hadj[5]); yw = f2_fma(h[5], v[1], yw); \
      hadj[6] = f2_fma(R, v[2], hadj[6]); yw = f2_fma(h[6], v[2], yw); \
      hadj[7] = f2_fma(R, v[3], hadj[7]); yw = f2_fma(h[7], v[3], yw); \
      hadj[8] = f2_fma(R, v[4], hadj[8]); yw = f2_fma(h[8], v[4], yw); \
      radial = f2_fma(dR, yw, radial); \
    } \
      f[9] = f2_sum(ang[0]); f[10] = f2_sum(ang[1]); f[11] = f2_sum(ang[2]); f[12] = f2_sum(ang[3]); f[13] = f2_sum(ang[4]); f[14] = f2_sum(ang[5]); f[15] = f2_sum(ang[6]); \
    }
#define SXB_S2_L1_ADJOINT_ROWS \
    TERM(0, 0, 0) \
    TERM(1, 1, 4) \
    TERM(2, 2, 9) \
    TERM(3, 3, 14) \
    TERM(4, 4, 21) \
    TERM(5, 5, 26) \
    TERM(6, 6, 31) \
    TERM(7, 7, 36) STORE(0) \
    TERM(0, 8, 41) \
    TERM(1, 10, 1) \
    TERM(2, 29, 1) \
    TERM(3, 43, 1) \
    TERM(4, 9, 3) \
    TERM(5, 27, 8) \
    TERM(6, 40, 13) \
    TERM(7, 15, 16) STORE(1) \
    TERM(0, 18, 11) \
    TERM(1, 21, 6) \
    TERM(2, 24, 6) \
    TERM(3, 33, 6) \
    TERM(4, 35, 11) \
    TERM(5, 37, 16) \
    TERM(6, 46, 6) \
    TERM(7, 50, 16) STORE(2) \
    TERM(0, 52, 11) \
    TERM(1, 55, 16) \
    TERM(2, 11, 29) TERM_ADD(2, 12, 39) \
    TERM(3, 13, 24) \
    TERM(4, 14, 19) \
    TERM(5, 28, 24) \
    TERM(6, 30, 29) \
    TERM(7, 31, 34) STORE(3) \
    TERM(0, 41, 19) \
    TERM(1, 42, 34) \
    TERM(2, 44, 29) TERM_ADD(2, 45, 39) \
    TERM(3, 16, 61) TERM_ADD(3, 17, 69) \
    TERM(4, 19, 57) TERM_ADD(4, 20, 65) \
    TERM(5, 22, 53) \
    TERM(6, 23, 49) \
    TERM(7, 25, 45) TERM_ADD(7, 26, 53) STORE(4) \
    TERM(0, 32, 49) \
    TERM(1, 34, 53) \
    TERM(2, 36, 57) \
    TERM(3, 38, 61) \
    TERM(4, 39, 65) \
    TERM(5, 47, 45) TERM_ADD(5, 48, 53) \
    TERM(6, 49, 49) \
    TERM(7, 51, 61) STORE(5) \
    TERM(0, 53, 57) TERM_ADD(0, 54, 65) \
    TERM(1, 56, 61) TERM_ADD(1, 57, 69) \
    TERM(2, 66, 2) \
    TERM(3, 79, 2) \
    TERM(4, 94, 2) \
    TERM(5, 108, 2) \
    TERM(6, 123, 2) \
    TERM(7, 59, 15) STORE(6) \
    TERM(0, 63, 5) \
    TERM(1, 72, 10) \
    TERM(2, 75, 5) \
    TERM(3, 86, 5) \
    TERM(4, 88, 10) \
    TERM(5, 90, 15) \
    TERM(6, 100, 15) \
    TERM(7, 102, 10) STORE(7) \
    TERM(0, 113, 5) \
    TERM(1, 117, 15) \
    TERM(2, 58, 18) \
    TERM(3, 71, 23) \
    TERM(4, 85, 28) \
    TERM(5, 98, 33) \
    TERM(6, 112, 38) \
    TERM(7, 67, 32) STORE(8) \
    TERM(0, 68, 37) \
    TERM(1, 69, 22) \
    TERM(2, 70, 27) \
    TERM(3, 78, 37) \
    TERM(4, 80, 32) TERM_ADD(4, 81, 42) \
    TERM(5, 82, 27) \
    TERM(6, 83, 22) \
    TERM(7, 84, 27) STORE(9) \
    TERM(0, 92, 22) \
    TERM(1, 93, 27) \
    TERM(2, 95, 32) \
    TERM(3, 96, 37) \
    TERM(4, 97, 42) \
    TERM(5, 105, 27) \
    TERM(6, 106, 22) \
    TERM(7, 107, 37) STORE(10) \
    TERM(0, 109, 32) TERM_ADD(0, 110, 42) \
    TERM(1, 111, 37) \
    TERM(2, 120, 27) \
    TERM(3, 121, 42) \
    TERM(4, 122, 37) \
    TERM(5, 124, 32) \
    TERM(6, 60, 60) TERM_ADD(6, 61, 68) \
    TERM(7, 62, 48) STORE(11) \
    TERM(0, 64, 44) TERM_ADD(0, 65, 52) \
    TERM(1, 73, 56) TERM_ADD(1, 74, 64) \
    TERM(2, 76, 52) \
    TERM(3, 77, 48) \
    TERM(4, 87, 52) \
    TERM(5, 89, 56) \
    TERM(6, 91, 60) \
    TERM(7, 99, 48) STORE(12) \
    TERM(0, 101, 60) \
    TERM(1, 103, 56) TERM_ADD(1, 104, 64) \
    TERM(2, 114, 44) TERM_ADD(2, 115, 52) \
    TERM(3, 116, 64) \
    TERM(4, 118, 60) TERM_ADD(4, 119, 68) \
    TERM(5, 128, 17) \
    TERM(6, 133, 7) \
    TERM(7, 139, 12) STORE(13) \
    TERM(0, 141, 17) \
    TERM(1, 144, 7) \
    TERM(2, 152, 17) \
    TERM(3, 155, 12) \
    TERM(4, 158, 7) \
    TERM(5, 161, 7) \
    TERM(6, 169, 7) \
    TERM(7, 171, 12) STORE(14) \
    TERM(0, 173, 17) \
    TERM(1, 181, 7) \
    TERM(2, 185, 17) \
    TERM(3, 187, 12) \
    TERM(4, 190, 17) \
    TERM(5, 197, 7) \
    TERM(6, 200, 17) \
    TERM(7, 203, 12) STORE(15) \
    TERM(0, 208, 7) \
    TERM(1, 213, 17) \
    TERM(2, 126, 40) \
    TERM(3, 127, 20) \
    TERM(4, 136, 35) \
    TERM(5, 137, 20) \
    TERM(6, 138, 25) \
    TERM(7, 148, 30) TERM_ADD(7, 149, 40) STORE(16) \
    TERM(0, 150, 25) \
    TERM(1, 151, 20) \
    TERM(2, 165, 25) \
    TERM(3, 166, 30) \
    TERM(4, 167, 35) \
    TERM(5, 177, 20) \
    TERM(6, 178, 35) \
    TERM(7, 179, 30) TERM_ADD(7, 180, 40) STORE(17) \
    TERM(0, 194, 25) \
    TERM(1, 195, 40) \
    TERM(2, 196, 35) \
    TERM(3, 206, 20) \
    TERM(4, 207, 40) \
    TERM(5, 125, 43) \
    TERM(6, 135, 47) \
    TERM(7, 147, 51) STORE(18) \
    TERM(0, 164, 55) \
    TERM(1, 176, 59) \
    TERM(2, 193, 63) \
    TERM(3, 205, 67) \
    TERM(4, 129, 62) \
    TERM(5, 130, 66) \
    TERM(6, 131, 46) \
    TERM(7, 132, 50) STORE(19) \
    TERM(0, 134, 54) \
    TERM(1, 140, 58) \
    TERM(2, 142, 62) TERM_ADD(2, 143, 70) \
    TERM(3, 145, 46) TERM_ADD(3, 146, 54) \
    TERM(4, 153, 62) TERM_ADD(4, 154, 70) \
    TERM(5, 156, 58) TERM_ADD(5, 157, 66) \
    TERM(6, 159, 54) \
    TERM(7, 160, 50) STORE(20) \
    TERM(0, 162, 46) TERM_ADD(0, 163, 54) \
    TERM(1, 168, 50) \
    TERM(2, 170, 54) \
    TERM(3, 172, 58) \
    TERM(4, 174, 62) \
    TERM(5, 175, 66) \
    TERM(6, 182, 46) TERM_ADD(6, 183, 54) \
    TERM(7, 184, 50) STORE(21) \
    TERM(0, 186, 62) \
    TERM(1, 188, 58) TERM_ADD(1, 189, 66) \
    TERM(2, 191, 62) TERM_ADD(2, 192, 70) \
    TERM(3, 198, 46) TERM_ADD(3, 199, 54) \
    TERM(4, 201, 62) TERM_ADD(4, 202, 70) \
    TERM(5, 204, 58) \
    TERM(6, 209, 54) \
    TERM(7, 210, 50) STORE(22) \
    TERM(0, 211, 70) \
    TERM(1, 212, 66) \
    TERM(2, 214, 62) \
    v[3] = 0ull; \
    v[4] = 0ull; \
    v[5] = 0ull; \
    v[6] = 0ull; \
    v[7] = 0ull; STORE(23)
#define SXB_S2_NUM_GROUPS 3
#define SXB_S2_G0_NUM_PATHS 10
#define SXB_S2_G0_NUM_ROWS 88
#define SXB_S2_G0_NUM_LME 40
#define SXB_S2_G0_PATH_LIST {0, 1, 3, 4, 5, 8, 9, 10, 13, 14}
#define SXB_S2_G0_LME_LIST {0, 1, 3, 4, 5, 8, 9, 10, 13, 14, 15, 18, 19, 20, 23, 24, 25, 28, 29, 30, 33, 34, 35, 38, 39, 40, 43, 44, 47, 48, 51, 52, 55, 56, 59, 60, 63, 64, 67, 68}
#define SXB_S2_G0_SOURCE_MASK 15u   // source components lm2 the set touches
// X(term, row inside the set, output inside the set)
#define SXB_S2_G0_TERMS(X) \
    X(0, 0, 0) \
    X(1, 13, 3) \
    X(2, 14, 6) \
    X(3, 15, 9) \
    X(9, 10, 2) \
    X(10, 1, 1) \
    X(11, 36, 18) \
    X(12, 36, 24) \
    X(13, 37, 15) \
    X(14, 38, 12) \
    X(27, 11, 5) \
    X(28, 39, 15) \
    X(29, 5, 1) \
    X(30, 40, 18) \
    X(31, 41, 21) \
    X(40, 12, 8) \
    X(41, 42, 12) \
    X(42, 43, 21) \
    X(43, 9, 1) \
    X(44, 44, 18) \
    X(45, 44, 24) \
    X(58, 31, 11) \
    X(59, 16, 10) \
    X(60, 73, 35) \
    X(61, 73, 39) \
    X(62, 74, 29) \
    X(63, 18, 4) \
    X(64, 75, 27) \
    X(65, 75, 31) \
    X(71, 32, 14) \
    X(72, 19, 7) \
    X(73, 76, 33) \
    X(74, 76, 37) \
    X(75, 20, 4) \
    X(76, 77, 31) \
    X(77, 78, 29) \
    X(85, 33, 17) \
    X(86, 22, 4) \
    X(87, 79, 31) \
    X(88, 23, 7) \
    X(89, 80, 33) \
    X(90, 24, 10) \
    X(91, 81, 35) \
    X(98, 34, 20) \
    X(99, 82, 29) \
    X(100, 26, 10) \
    X(101, 83, 35) \
    X(102, 27, 7) \
    X(103, 84, 33) \
    X(104, 84, 37) \
    X(112, 35, 23) \
    X(113, 28, 4) \
    X(114, 85, 27) \
    X(115, 85, 31) \
    X(116, 86, 37) \
    X(117, 30, 10) \
    X(118, 87, 35) \
    X(119, 87, 39) \
    X(125, 66, 26) \
    X(126, 45, 25) \
    X(127, 47, 13) \
    X(135, 67, 28) \
    X(136, 48, 22) \
    X(137, 49, 13) \
    X(138, 50, 16) \
    X(147, 68, 30) \
    X(148, 51, 19) \
    X(149, 51, 25) \
    X(150, 52, 16) \
    X(151, 53, 13) \
    X(164, 69, 32) \
    X(165, 54, 16) \
    X(166, 55, 19) \
    X(167, 56, 22) \
    X(176, 70, 34) \
    X(177, 57, 13) \
    X(178, 58, 22) \
    X(179, 59, 19) \
    X(180, 59, 25) \
    X(193, 71, 36) \
    X(194, 60, 16) \
    X(195, 61, 25) \
    X(196, 62, 22) \
    X(205, 72, 38) \
    X(206, 63, 13) \
    X(207, 65, 25)
#define SXB_S2_G0_FORWARD_BODY \
    { /* path 0: edge l=0, source l=0 -> l=0 */ \
      const float t0 = R[0] * h[0]; \
      acc[0] = fmaf(t0, y[0], acc[0]); \
    } \
    { /* path 1: edge l=1, source l=1 -> l=0 */ \
      const float t0 = R[1] * h[1]; \
      const float t1 = R[1] * h[2]; \
      const float t2 = R[1] * h[3]; \
      acc[1] = fmaf(t0, y[1], acc[1]); \
      acc[2] = fmaf(t1, y[1], acc[2]); \
      acc[3] = fmaf(t2, y[1], acc[3]); \
      acc[4] = fmaf(t0, y[2], acc[4]); \
      acc[5] = fmaf(t1, y[2], acc[5]); \
      acc[6] = fmaf(t2, y[2], acc[6]); \
      acc[7] = fmaf(t0, y[3], acc[7]); \
      acc[8] = fmaf(t1, y[3], acc[8]); \
      acc[9] = fmaf(t2, y[3], acc[9]); \
    } \
    { /* path 3: edge l=1, source l=0 -> l=1 */ \
      const float t0 = R[2] * h[0]; \
      acc[10] = fmaf(t0, y[1], acc[10]); \
      acc[11] = fmaf(t0, y[2], acc[11]); \
      acc[12] = fmaf(t0, y[3], acc[12]); \
    } \
    { /* path 4: edge l=0, source l=1 -> l=1 */ \
      const float t0 = R[3] * h[1]; \
      const float t1 = R[3] * h[2]; \
      const float t2 = R[3] * h[3]; \
      acc[13] = fmaf(t0, y[0], acc[13]); \
      acc[14] = fmaf(t1, y[0], acc[14]); \
      acc[15] = fmaf(t2, y[0], acc[15]); \
    } \
    { /* path 5: edge l=2, source l=1 -> l=1 */ \
      const float t0 = R[4] * h[1]; \
      const float t1 = R[4] * h[2]; \
      const float t2 = R[4] * h[3]; \
      acc[16] = fmaf(t0, y[4], acc[16]); \
      acc[17] = fmaf(t1, y[4], acc[17]); \
      acc[18] = fmaf(t2, y[4], acc[18]); \
      acc[19] = fmaf(t0, y[5], acc[19]); \
      acc[20] = fmaf(t1, y[5], acc[20]); \
      acc[21] = fmaf(t2, y[5], acc[21]); \
      acc[22] = fmaf(t0, y[6], acc[22]); \
      acc[23] = fmaf(t1, y[6], acc[23]); \
      acc[24] = fmaf(t2, y[6], acc[24]); \
      acc[25] = fmaf(t0, y[7], acc[25]); \
      acc[26] = fmaf(t1, y[7], acc[26]); \
      acc[27] = fmaf(t2, y[7], acc[27]); \
      acc[28] = fmaf(t0, y[8], acc[28]); \
      acc[29] = fmaf(t1, y[8], acc[29]); \
      acc[30] = fmaf(t2, y[8], acc[30]); \
    } \
    { /* path 8: edge l=2, source l=0 -> l=2 */ \
      const float t0 = R[5] * h[0]; \
      acc[31] = fmaf(t0, y[4], acc[31]); \
      acc[32] = fmaf(t0, y[5], acc[32]); \
      acc[33] = fmaf(t0, y[6], acc[33]); \
      acc[34] = fmaf(t0, y[7], acc[34]); \
      acc[35] = fmaf(t0, y[8], acc[35]); \
    } \
    { /* path 9: edge l=1, source l=1 -> l=2 */ \
      const float t0 = R[6] * h[1]; \
      const float t1 = R[6] * h[2]; \
      const float t2 = R[6] * h[3]; \
      acc[36] = fmaf(t0, y[1], acc[36]); \
      acc[37] = fmaf(t1, y[1], acc[37]); \
      acc[38] = fmaf(t2, y[1], acc[38]); \
      acc[39] = fmaf(t0, y[2], acc[39]); \
      acc[40] = fmaf(t1, y[2], acc[40]); \
      acc[41] = fmaf(t2, y[2], acc[41]); \
      acc[42] = fmaf(t0, y[3], acc[42]); \
      acc[43] = fmaf(t1, y[3], acc[43]); \
      acc[44] = fmaf(t2, y[3], acc[44]); \
    } \
    { /* path 10: edge l=3, source l=1 -> l=2 */ \
      const float t0 = R[7] * h[1]; \
      const float t1 = R[7] * h[2]; \
      const float t2 = R[7] * h[3]; \
      acc[45] = fmaf(t0, y[9], acc[45]); \
      acc[46] = fmaf(t1, y[9], acc[46]); \
      acc[47] = fmaf(t2, y[9], acc[47]); \
      acc[48] = fmaf(t0, y[10], acc[48]); \
      acc[49] = fmaf(t1, y[10], acc[49]); \
      acc[50] = fmaf(t2, y[10], acc[50]); \
      acc[51] = fmaf(t0, y[11], acc[51]); \
      acc[52] = fmaf(t1, y[11], acc[52]); \
      acc[53] = fmaf(t2, y[11], acc[53]); \
      acc[54] = fmaf(t0, y[12], acc[54]); \
      acc[55] = fmaf(t1, y[12], acc[55]); \
      acc[56] = fmaf(t2, y[12], acc[56]); \
      acc[57] = fmaf(t0, y[13], acc[57]); \
      acc[58] = fmaf(t1, y[13], acc[58]); \
      acc[59] = fmaf(t2, y[13], acc[59]); \
      acc[60] = fmaf(t0, y[14], acc[60]); \
      acc[61] = fmaf(t1, y[14], acc[61]); \
      acc[62] = fmaf(t2, y[14], acc[62]); \
      acc[63] = fmaf(t0, y[15], acc[63]); \
      acc[64] = fmaf(t1, y[15], acc[64]); \
      acc[65] = fmaf(t2, y[15], acc[65]); \
    } \
    { /* path 13: edge l=3, source l=0 -> l=3 */ \
      const float t0 = R[8] * h[0]; \
      acc[66] = fmaf(t0, y[9], acc[66]); \
      acc[67] = fmaf(t0, y[10], acc[67]); \
      acc[68] = fmaf(t0, y[11], acc[68]); \
      acc[69] = fmaf(t0, y[12], acc[69]); \
      acc[70] = fmaf(t0, y[13], acc[70]); \
      acc[71] = fmaf(t0, y[14], acc[71]); \
      acc[72] = fmaf(t0, y[15], acc[72]); \
    } \
    { /* path 14: edge l=2, source l=1 -> l=3 */ \
      const float t0 = R[9] * h[1]; \
      const float t1 = R[9] * h[2]; \
      const float t2 = R[9] * h[3]; \
      acc[73] = fmaf(t0, y[4], acc[73]); \
      acc[74] = fmaf(t1, y[4], acc[74]); \
      acc[75] = fmaf(t2, y[4], acc[75]); \
      acc[76] = fmaf(t0, y[5], acc[76]); \
      acc[77] = fmaf(t1, y[5], acc[77]); \
      acc[78] = fmaf(t2, y[5], acc[78]); \
      acc[79] = fmaf(t0, y[6], acc[79]); \
      acc[80] = fmaf(t1, y[6], acc[80]); \
      acc[81] = fmaf(t2, y[6], acc[81]); \
      acc[82] = fmaf(t0, y[7], acc[82]); \
      acc[83] = fmaf(t1, y[7], acc[83]); \
      acc[84] = fmaf(t2, y[7], acc[84]); \
      acc[85] = fmaf(t0, y[8], acc[85]); \
      acc[86] = fmaf(t1, y[8], acc[86]); \
      acc[87] = fmaf(t2, y[8], acc[87]); \
    }
#define SXB_S2_G1_NUM_PATHS 4
#define SXB_S2_G1_NUM_ROWS 80
#define SXB_S2_G1_NUM_LME 12
#define SXB_S2_G1_PATH_LIST {2, 6, 7, 11}
#define SXB_S2_G1_LME_LIST {2, 6, 7, 11, 12, 16, 17, 21, 26, 31, 36, 41}
#define SXB_S2_G1_SOURCE_MASK 496u   // source components lm2 the set touches
// X(term, row inside the set, output inside the set)
#define SXB_S2_G1_TERMS(X) \
    X(4, 75, 7) \
    X(5, 76, 8) \
    X(6, 77, 9) \
    X(7, 78, 10) \
    X(8, 79, 11) \
    X(15, 25, 5) \
    X(18, 26, 3) \
    X(21, 27, 1) \
    X(24, 29, 1) \
    X(33, 31, 1) \
    X(35, 32, 3) \
    X(37, 33, 5) \
    X(46, 35, 1) \
    X(50, 37, 5) \
    X(52, 38, 3) \
    X(55, 39, 5) \
    X(66, 0, 0) \
    X(79, 6, 0) \
    X(94, 12, 0) \
    X(108, 18, 0) \
    X(123, 24, 0) \
    X(128, 40, 6) \
    X(133, 44, 2) \
    X(139, 45, 4) \
    X(141, 46, 6) \
    X(144, 48, 2) \
    X(152, 50, 6) \
    X(155, 51, 4) \
    X(158, 52, 2) \
    X(161, 54, 2) \
    X(169, 56, 2) \
    X(171, 57, 4) \
    X(173, 58, 6) \
    X(181, 60, 2) \
    X(185, 62, 6) \
    X(187, 63, 4) \
    X(190, 64, 6) \
    X(197, 66, 2) \
    X(200, 68, 6) \
    X(203, 69, 4) \
    X(208, 70, 2) \
    X(213, 74, 6)
#define SXB_S2_G1_FORWARD_BODY \
    { /* path 2: edge l=2, source l=2 -> l=0 */ \
      const float t0 = R[0] * h[4]; \
      const float t1 = R[0] * h[5]; \
      const float t2 = R[0] * h[6]; \
      const float t3 = R[0] * h[7]; \
      const float t4 = R[0] * h[8]; \
      acc[0] = fmaf(t0, y[4], acc[0]); \
      acc[1] = fmaf(t1, y[4], acc[1]); \
      acc[2] = fmaf(t2, y[4], acc[2]); \
      acc[3] = fmaf(t3, y[4], acc[3]); \
      acc[4] = fmaf(t4, y[4], acc[4]); \
      acc[5] = fmaf(t0, y[5], acc[5]); \
      acc[6] = fmaf(t1, y[5], acc[6]); \
      acc[7] = fmaf(t2, y[5], acc[7]); \
      acc[8] = fmaf(t3, y[5], acc[8]); \
      acc[9] = fmaf(t4, y[5], acc[9]); \
      acc[10] = fmaf(t0, y[6], acc[10]); \
      acc[11] = fmaf(t1, y[6], acc[11]); \
      acc[12] = fmaf(t2, y[6], acc[12]); \
      acc[13] = fmaf(t3, y[6], acc[13]); \
      acc[14] = fmaf(t4, y[6], acc[14]); \
      acc[15] = fmaf(t0, y[7], acc[15]); \
      acc[16] = fmaf(t1, y[7], acc[16]); \
      acc[17] = fmaf(t2, y[7], acc[17]); \
      acc[18] = fmaf(t3, y[7], acc[18]); \
      acc[19] = fmaf(t4, y[7], acc[19]); \
      acc[20] = fmaf(t0, y[8], acc[20]); \
      acc[21] = fmaf(t1, y[8], acc[21]); \
      acc[22] = fmaf(t2, y[8], acc[22]); \
      acc[23] = fmaf(t3, y[8], acc[23]); \
      acc[24] = fmaf(t4, y[8], acc[24]); \
    } \
    { /* path 6: edge l=1, source l=2 -> l=1 */ \
      const float t0 = R[1] * h[4]; \
      const float t1 = R[1] * h[5]; \
      const float t2 = R[1] * h[6]; \
      const float t3 = R[1] * h[7]; \
      const float t4 = R[1] * h[8]; \
      acc[25] = fmaf(t0, y[1], acc[25]); \
      acc[26] = fmaf(t1, y[1], acc[26]); \
      acc[27] = fmaf(t2, y[1], acc[27]); \
      acc[28] = fmaf(t3, y[1], acc[28]); \
      acc[29] = fmaf(t4, y[1], acc[29]); \
      acc[30] = fmaf(t0, y[2], acc[30]); \
      acc[31] = fmaf(t1, y[2], acc[31]); \
      acc[32] = fmaf(t2, y[2], acc[32]); \
      acc[33] = fmaf(t3, y[2], acc[33]); \
      acc[34] = fmaf(t4, y[2], acc[34]); \
      acc[35] = fmaf(t0, y[3], acc[35]); \
      acc[36] = fmaf(t1, y[3], acc[36]); \
      acc[37] = fmaf(t2, y[3], acc[37]); \
      acc[38] = fmaf(t3, y[3], acc[38]); \
      acc[39] = fmaf(t4, y[3], acc[39]); \
    } \
    { /* path 7: edge l=3, source l=2 -> l=1 */ \
      const float t0 = R[2] * h[4]; \
      const float t1 = R[2] * h[5]; \
      const float t2 = R[2] * h[6]; \
      const float t3 = R[2] * h[7]; \
      const float t4 = R[2] * h[8]; \
      acc[40] = fmaf(t0, y[9], acc[40]); \
      acc[41] = fmaf(t1, y[9], acc[41]); \
      acc[42] = fmaf(t2, y[9], acc[42]); \
      acc[43] = fmaf(t3, y[9], acc[43]); \
      acc[44] = fmaf(t4, y[9], acc[44]); \
      acc[45] = fmaf(t0, y[10], acc[45]); \
      acc[46] = fmaf(t1, y[10], acc[46]); \
      acc[47] = fmaf(t2, y[10], acc[47]); \
      acc[48] = fmaf(t3, y[10], acc[48]); \
      acc[49] = fmaf(t4, y[10], acc[49]); \
      acc[50] = fmaf(t0, y[11], acc[50]); \
      acc[51] = fmaf(t1, y[11], acc[51]); \
      acc[52] = fmaf(t2, y[11], acc[52]); \
      acc[53] = fmaf(t3, y[11], acc[53]); \
      acc[54] = fmaf(t4, y[11], acc[54]); \
      acc[55] = fmaf(t0, y[12], acc[55]); \
      acc[56] = fmaf(t1, y[12], acc[56]); \
      acc[57] = fmaf(t2, y[12], acc[57]); \
      acc[58] = fmaf(t3, y[12], acc[58]); \
      acc[59] = fmaf(t4, y[12], acc[59]); \
      acc[60] = fmaf(t0, y[13], acc[60]); \
      acc[61] = fmaf(t1, y[13], acc[61]); \
      acc[62] = fmaf(t2, y[13], acc[62]); \
      acc[63] = fmaf(t3, y[13], acc[63]); \
      acc[64] = fmaf(t4, y[13], acc[64]); \
      acc[65] = fmaf(t0, y[14], acc[65]); \
      acc[66] = fmaf(t1, y[14], acc[66]); \
      acc[67] = fmaf(t2, y[14], acc[67]); \
      acc[68] = fmaf(t3, y[14], acc[68]); \
      acc[69] = fmaf(t4, y[14], acc[69]); \
      acc[70] = fmaf(t0, y[15], acc[70]); \
      acc[71] = fmaf(t1, y[15], acc[71]); \
      acc[72] = fmaf(t2, y[15], acc[72]); \
      acc[73] = fmaf(t3, y[15], acc[73]); \
      acc[74] = fmaf(t4, y[15], acc[74]); \
    } \
    { /* path 11: edge l=0, source l=2 -> l=2 */ \
      const float t0 = R[3] * h[4]; \
      const float t1 = R[3] * h[5]; \
      const float t2 = R[3] * h[6]; \
      const float t3 = R[3] * h[7]; \
      const float t4 = R[3] * h[8]; \
      acc[75] = fmaf(t0, y[0], acc[75]); \
      acc[76] = fmaf(t1, y[0], acc[76]); \
      acc[77] = fmaf(t2, y[0], acc[77]); \
      acc[78] = fmaf(t3, y[0], acc[78]); \
      acc[79] = fmaf(t4, y[0], acc[79]); \
    }
#define SXB_S2_G2_NUM_PATHS 3
#define SXB_S2_G2_NUM_ROWS 75
#define SXB_S2_G2_NUM_LME 19
#define SXB_S2_G2_PATH_LIST {12, 15, 16}
#define SXB_S2_G2_LME_LIST {22, 27, 32, 37, 42, 45, 46, 49, 50, 53, 54, 57, 58, 61, 62, 65, 66, 69, 70}
#define SXB_S2_G2_SOURCE_MASK 496u   // source components lm2 the set touches
// X(term, row inside the set, output inside the set)
#define SXB_S2_G2_TERMS(X) \
    X(16, 25, 13) \
    X(17, 25, 17) \
    X(19, 26, 11) \
    X(20, 26, 15) \
    X(22, 27, 9) \
    X(23, 28, 7) \
    X(25, 29, 5) \
    X(26, 29, 9) \
    X(32, 30, 7) \
    X(34, 31, 9) \
    X(36, 32, 11) \
    X(38, 33, 13) \
    X(39, 34, 15) \
    X(47, 35, 5) \
    X(48, 35, 9) \
    X(49, 36, 7) \
    X(51, 37, 13) \
    X(53, 38, 11) \
    X(54, 38, 15) \
    X(56, 39, 13) \
    X(57, 39, 17) \
    X(67, 0, 2) \
    X(68, 1, 3) \
    X(69, 2, 0) \
    X(70, 3, 1) \
    X(78, 5, 3) \
    X(80, 6, 2) \
    X(81, 6, 4) \
    X(82, 7, 1) \
    X(83, 8, 0) \
    X(84, 9, 1) \
    X(92, 10, 0) \
    X(93, 11, 1) \
    X(95, 12, 2) \
    X(96, 13, 3) \
    X(97, 14, 4) \
    X(105, 15, 1) \
    X(106, 16, 0) \
    X(107, 17, 3) \
    X(109, 18, 2) \
    X(110, 18, 4) \
    X(111, 19, 3) \
    X(120, 21, 1) \
    X(121, 22, 4) \
    X(122, 23, 3) \
    X(124, 24, 2) \
    X(129, 40, 14) \
    X(130, 41, 16) \
    X(131, 42, 6) \
    X(132, 43, 8) \
    X(134, 44, 10) \
    X(140, 45, 12) \
    X(142, 46, 14) \
    X(143, 46, 18) \
    X(145, 48, 6) \
    X(146, 48, 10) \
    X(153, 50, 14) \
    X(154, 50, 18) \
    X(156, 51, 12) \
    X(157, 51, 16) \
    X(159, 52, 10) \
    X(160, 53, 8) \
    X(162, 54, 6) \
    X(163, 54, 10) \
    X(168, 55, 8) \
    X(170, 56, 10) \
    X(172, 57, 12) \
    X(174, 58, 14) \
    X(175, 59, 16) \
    X(182, 60, 6) \
    X(183, 60, 10) \
    X(184, 61, 8) \
    X(186, 62, 14) \
    X(188, 63, 12) \
    X(189, 63, 16) \
    X(191, 64, 14) \
    X(192, 64, 18) \
    X(198, 66, 6) \
    X(199, 66, 10) \
    X(201, 68, 14) \
    X(202, 68, 18) \
    X(204, 69, 12) \
    X(209, 70, 10) \
    X(210, 71, 8) \
    X(211, 72, 18) \
    X(212, 73, 16) \
    X(214, 74, 14)
#define SXB_S2_G2_FORWARD_BODY \
    { /* path 12: edge l=2, source l=2 -> l=2 */ \
      const float t0 = R[0] * h[4]; \
      const float t1 = R[0] * h[5]; \
      const float t2 = R[0] * h[6]; \
      const float t3 = R[0] * h[7]; \
      const float t4 = R[0] * h[8]; \
      acc[0] = fmaf(t0, y[4], acc[0]); \
      acc[1] = fmaf(t1, y[4], acc[1]); \
      acc[2] = fmaf(t2, y[4], acc[2]); \
      acc[3] = fmaf(t3, y[4], acc[3]); \
      acc[4] = fmaf(t4, y[4], acc[4]); \
      acc[5] = fmaf(t0, y[5], acc[5]); \
      acc[6] = fmaf(t1, y[5], acc[6]); \
      acc[7] = fmaf(t2, y[5], acc[7]); \
      acc[8] = fmaf(t3, y[5], acc[8]); \
      acc[9] = fmaf(t4, y[5], acc[9]); \
      acc[10] = fmaf(t0, y[6], acc[10]); \
      acc[11] = fmaf(t1, y[6], acc[11]); \
      acc[12] = fmaf(t2, y[6], acc[12]); \
      acc[13] = fmaf(t3, y[6], acc[13]); \
      acc[14] = fmaf(t4, y[6], acc[14]); \
      acc[15] = fmaf(t0, y[7], acc[15]); \
      acc[16] = fmaf(t1, y[7], acc[16]); \
      acc[17] = fmaf(t2, y[7], acc[17]); \
      acc[18] = fmaf(t3, y[7], acc[18]); \
      acc[19] = fmaf(t4, y[7], acc[19]); \
      acc[20] = fmaf(t0, y[8], acc[20]); \
      acc[21] = fmaf(t1, y[8], acc[21]); \
      acc[22] = fmaf(t2, y[8], acc[22]); \
      acc[23] = fmaf(t3, y[8], acc[23]); \
      acc[24] = fmaf(t4, y[8], acc[24]); \
    } \
    { /* path 15: edge l=1, source l=2 -> l=3 */ \
      const float t0 = R[1] * h[4]; \
      const float t1 = R[1] * h[5]; \
      const float t2 = R[1] * h[6]; \
      const float t3 = R[1] * h[7]; \
      const float t4 = R[1] * h[8]; \
      acc[25] = fmaf(t0, y[1], acc[25]); \
      acc[26] = fmaf(t1, y[1], acc[26]); \
      acc[27] = fmaf(t2, y[1], acc[27]); \
      acc[28] = fmaf(t3, y[1], acc[28]); \
      acc[29] = fmaf(t4, y[1], acc[29]); \
      acc[30] = fmaf(t0, y[2], acc[30]); \
      acc[31] = fmaf(t1, y[2], acc[31]); \
      acc[32] = fmaf(t2, y[2], acc[32]); \
      acc[33] = fmaf(t3, y[2], acc[33]); \
      acc[34] = fmaf(t4, y[2], acc[34]); \
      acc[35] = fmaf(t0, y[3], acc[35]); \
      acc[36] = fmaf(t1, y[3], acc[36]); \
      acc[37] = fmaf(t2, y[3], acc[37]); \
      acc[38] = fmaf(t3, y[3], acc[38]); \
      acc[39] = fmaf(t4, y[3], acc[39]); \
    } \
    { /* path 16: edge l=3, source l=2 -> l=3 */ \
      const float t0 = R[2] * h[4]; \
      const float t1 = R[2] * h[5]; \
      const float t2 = R[2] * h[6]; \
      const float t3 = R[2] * h[7]; \
      const float t4 = R[2] * h[8]; \
      acc[40] = fmaf(t0, y[9], acc[40]); \
      acc[41] = fmaf(t1, y[9], acc[41]); \
      acc[42] = fmaf(t2, y[9], acc[42]); \
      acc[43] = fmaf(t3, y[9], acc[43]); \
      acc[44] = fmaf(t4, y[9], acc[44]); \
      acc[45] = fmaf(t0, y[10], acc[45]); \
      acc[46] = fmaf(t1, y[10], acc[46]); \
      acc[47] = fmaf(t2, y[10], acc[47]); \
      acc[48] = fmaf(t3, y[10], acc[48]); \
      acc[49] = fmaf(t4, y[10], acc[49]); \
      acc[50] = fmaf(t0, y[11], acc[50]); \
      acc[51] = fmaf(t1, y[11], acc[51]); \
      acc[52] = fmaf(t2, y[11], acc[52]); \
      acc[53] = fmaf(t3, y[11], acc[53]); \
      acc[54] = fmaf(t4, y[11], acc[54]); \
      acc[55] = fmaf(t0, y[12], acc[55]); \
      acc[56] = fmaf(t1, y[12], acc[56]); \
      acc[57] = fmaf(t2, y[12], acc[57]); \
      acc[58] = fmaf(t3, y[12], acc[58]); \
      acc[59] = fmaf(t4, y[12], acc[59]); \
      acc[60] = fmaf(t0, y[13], acc[60]); \
      acc[61] = fmaf(t1, y[13], acc[61]); \
      acc[62] = fmaf(t2, y[13], acc[62]); \
      acc[63] = fmaf(t3, y[13], acc[63]); \
      acc[64] = fmaf(t4, y[13], acc[64]); \
      acc[65] = fmaf(t0, y[14], acc[65]); \
      acc[66] = fmaf(t1, y[14], acc[66]); \
      acc[67] = fmaf(t2, y[14], acc[67]); \
      acc[68] = fmaf(t3, y[14], acc[68]); \
      acc[69] = fmaf(t4, y[14], acc[69]); \
      acc[70] = fmaf(t0, y[15], acc[70]); \
      acc[71] = fmaf(t1, y[15], acc[71]); \
      acc[72] = fmaf(t2, y[15], acc[72]); \
      acc[73] = fmaf(t3, y[15], acc[73]); \
      acc[74] = fmaf(t4, y[15], acc[74]); \
    }
