// fs_rng.cuh -- device random number generators, bit-identical to the reference's.
//
// Included into every NVRTC module built by fs_api.cu (kept free of host headers).
//
//  * xorshift128 exactly as FeynSimul/GPUsrc/kernel.c:214-239: float = float(w) * 2^-32
//    (the constant 2.328306437080797e-10 is 2^-32 once rounded to FP32, which is what the
//    reference's -cl-single-precision-constant build uses).
//  * RANLUX in the RANLUXCL v1.3.1 formulation the reference vendors
//    (examples/pyopencl-ranluxcl.cl): subtract-with-borrow on 24 lags with the p-skip
//    schedule, xorshift64 seeding and 32-cycle warm-up.  The lags are multiples of 2^-24 in
//    [0, 1), so this file keeps them as 24-bit digits packed into 32-bit words and runs the
//    subtract-with-borrow as a hardware borrow chain (see FsRanlux); the results are
//    identical because every float operation of the reference on these values is exact.
//    Output floats are formed exactly as the reference forms them (small values get the
//    next lag's bits, zero maps to 2^-48).
//  * State tables in global memory keep the reference's 28-word float layout
//    (pyopencl-ranluxcl.cl:264-277), converted on load and store.
#pragma once

typedef unsigned int fs_u32;
typedef unsigned long long fs_u64;

// ---------------------------------------------------------------- xorshift128
struct FsXorshift {
    fs_u32 x, y, z, w;
};

__device__ __forceinline__ fs_u32 fs_xs_next(FsXorshift &s)
{
    fs_u32 t = s.x ^ (s.x << 11);
    s.x = s.y;
    s.y = s.z;
    s.z = s.w;
    s.w = s.w ^ (s.w >> 19) ^ (t ^ (t >> 8));
    return s.w;
}

__device__ __forceinline__ float fs_xs_float(FsXorshift &s)
{
    return __fmul_rn(__uint2float_rn(fs_xs_next(s)), 0x1p-32f);
}

__device__ __forceinline__ double fs_xs_double(FsXorshift &s)
{
    // ENABLE_DOUBLE build of kernel.c:229: double(w) * 2.328306437080797e-10 in FP64
    return __dmul_rn((double)fs_xs_next(s), 2.328306437080797e-10);
}

// ---------------------------------------------------------------- RANLUX
// The 24 lags (k for value k * 2^-24, 0 <= k < 2^24) are the base-2^24 digits of one 576-bit
// integer in 18 words, in the order the recurrence updates them: digit p at bits 24 p.  A step
// replaces digit p by (digit p - 10) - (digit p) - borrow (cyclically; the digits below p are
// already new), so consecutive steps are one long subtraction, whose borrows run through the
// words as through the digits: word j becomes M_j - w_j - borrow with the minuend M_j = the 32
// bits 240 below, i.e. the upper half of word j - 8 under the lower half of word j - 7.  A
// step costs 3/4 of a funnel shift and a `subc.cc`, 1.5 instructions (one digit per word
// takes a `subc.cc` and a mask, 2), on a chain of 18 dependent instructions a cycle instead
// of 24, in 18 registers instead of 24.
//
// The frame: digit 0 is where the next skip starts, so the 24 values between two skips are
// the digits 0..23 in order, four ("a quad", words 3 q .. 3 q + 2) per generator call, and
// every skip starts at digit 0.  A skip of 24 k + m steps moves the generator's position by
// m digits; the words are renamed (rotated) so that the position is digit 0 again, and `rot`
// keeps the table position of digit 0.
// The borrow enters a chain as `0 - c` and leaves it as `0 - 0 - borrow` (so c is 0 or
// 0xFFFFFFFF), i.e. only through subtractions, whichever polarity the flag has.
struct FsRanlux {
    fs_u32 w[18];
    fs_u32 carry;   // 0 or 0xFFFFFFFF (the reference stores 0 or 2^-24)
    fs_u32 q;       // next quad, 0..5
    fs_u32 rot;     // the reference's position (its stepnr) of digit 0
};

#define FS_RL_BORROW_IN(c) "{\n\t.reg .u32 fsz, fsm;\n\tmov.u32 fsz, 0;\n\tsub.cc.u32 fsz, fsz, " c ";\n\t"
#define FS_RL_STEP(w, lo, hi) "shf.l.wrap.b32 fsm, " lo ", " hi ", 16;\n\tsubc.cc.u32 " w ", fsm, " w ";\n\t"
#define FS_RL_BORROW_OUT(c) "mov.u32 fsz, 0;\n\tsubc.u32 " c ", fsz, fsz;\n\t}"

// Chains of one quad, of the runs of quads that next_12 draws, and of the whole cycle; a
// chain names only the words it reads or writes.
__device__ __forceinline__ void fs_rl_chain_q0(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%3")
        FS_RL_STEP("%0", "%4", "%5") FS_RL_STEP("%1", "%5", "%6") FS_RL_STEP("%2", "%6", "%7")
        FS_RL_BORROW_OUT("%3")
        : "+r"(r.w[0]), "+r"(r.w[1]), "+r"(r.w[2]), "+r"(r.carry)
        : "r"(r.w[10]), "r"(r.w[11]), "r"(r.w[12]), "r"(r.w[13]));
}

__device__ __forceinline__ void fs_rl_chain_q1(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%3")
        FS_RL_STEP("%0", "%4", "%5") FS_RL_STEP("%1", "%5", "%6") FS_RL_STEP("%2", "%6", "%7")
        FS_RL_BORROW_OUT("%3")
        : "+r"(r.w[3]), "+r"(r.w[4]), "+r"(r.w[5]), "+r"(r.carry)
        : "r"(r.w[13]), "r"(r.w[14]), "r"(r.w[15]), "r"(r.w[16]));
}

__device__ __forceinline__ void fs_rl_chain_q2(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%3")
        FS_RL_STEP("%0", "%6", "%7") FS_RL_STEP("%1", "%7", "%4") FS_RL_STEP("%2", "%4", "%5")
        FS_RL_BORROW_OUT("%3")
        : "+r"(r.w[6]), "+r"(r.w[7]), "+r"(r.w[8]), "+r"(r.carry)
        : "r"(r.w[0]), "r"(r.w[1]), "r"(r.w[16]), "r"(r.w[17]));
}

__device__ __forceinline__ void fs_rl_chain_q3(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%3")
        FS_RL_STEP("%0", "%4", "%5") FS_RL_STEP("%1", "%5", "%6") FS_RL_STEP("%2", "%6", "%7")
        FS_RL_BORROW_OUT("%3")
        : "+r"(r.w[9]), "+r"(r.w[10]), "+r"(r.w[11]), "+r"(r.carry)
        : "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[3]), "r"(r.w[4]));
}

__device__ __forceinline__ void fs_rl_chain_q4(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%3")
        FS_RL_STEP("%0", "%4", "%5") FS_RL_STEP("%1", "%5", "%6") FS_RL_STEP("%2", "%6", "%7")
        FS_RL_BORROW_OUT("%3")
        : "+r"(r.w[12]), "+r"(r.w[13]), "+r"(r.w[14]), "+r"(r.carry)
        : "r"(r.w[4]), "r"(r.w[5]), "r"(r.w[6]), "r"(r.w[7]));
}

__device__ __forceinline__ void fs_rl_chain_q5(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%3")
        FS_RL_STEP("%0", "%4", "%5") FS_RL_STEP("%1", "%5", "%6") FS_RL_STEP("%2", "%6", "%7")
        FS_RL_BORROW_OUT("%3")
        : "+r"(r.w[15]), "+r"(r.w[16]), "+r"(r.w[17]), "+r"(r.carry)
        : "r"(r.w[7]), "r"(r.w[8]), "r"(r.w[9]), "r"(r.w[10]));
}

__device__ __forceinline__ void fs_rl_chain_q01(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%6")
        FS_RL_STEP("%0", "%7", "%8") FS_RL_STEP("%1", "%8", "%9") FS_RL_STEP("%2", "%9", "%10")
        FS_RL_STEP("%3", "%10", "%11") FS_RL_STEP("%4", "%11", "%12") FS_RL_STEP("%5", "%12", "%13")
        FS_RL_BORROW_OUT("%6")
        : "+r"(r.w[0]), "+r"(r.w[1]), "+r"(r.w[2]), "+r"(r.w[3]), "+r"(r.w[4]), "+r"(r.w[5]),
          "+r"(r.carry)
        : "r"(r.w[10]), "r"(r.w[11]), "r"(r.w[12]), "r"(r.w[13]), "r"(r.w[14]), "r"(r.w[15]),
          "r"(r.w[16]));
}

__device__ __forceinline__ void fs_rl_chain_q45(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%6")
        FS_RL_STEP("%0", "%7", "%8") FS_RL_STEP("%1", "%8", "%9") FS_RL_STEP("%2", "%9", "%10")
        FS_RL_STEP("%3", "%10", "%11") FS_RL_STEP("%4", "%11", "%12") FS_RL_STEP("%5", "%12", "%13")
        FS_RL_BORROW_OUT("%6")
        : "+r"(r.w[12]), "+r"(r.w[13]), "+r"(r.w[14]), "+r"(r.w[15]), "+r"(r.w[16]),
          "+r"(r.w[17]), "+r"(r.carry)
        : "r"(r.w[4]), "r"(r.w[5]), "r"(r.w[6]), "r"(r.w[7]), "r"(r.w[8]), "r"(r.w[9]),
          "r"(r.w[10]));
}

__device__ __forceinline__ void fs_rl_chain_q012(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%9")
        FS_RL_STEP("%0", "%10", "%11") FS_RL_STEP("%1", "%11", "%12") FS_RL_STEP("%2", "%12", "%13")
        FS_RL_STEP("%3", "%13", "%14") FS_RL_STEP("%4", "%14", "%15") FS_RL_STEP("%5", "%15", "%16")
        FS_RL_STEP("%6", "%16", "%17") FS_RL_STEP("%7", "%17", "%0") FS_RL_STEP("%8", "%0", "%1")
        FS_RL_BORROW_OUT("%9")
        : "+r"(r.w[0]), "+r"(r.w[1]), "+r"(r.w[2]), "+r"(r.w[3]), "+r"(r.w[4]), "+r"(r.w[5]),
          "+r"(r.w[6]), "+r"(r.w[7]), "+r"(r.w[8]), "+r"(r.carry)
        : "r"(r.w[10]), "r"(r.w[11]), "r"(r.w[12]), "r"(r.w[13]), "r"(r.w[14]), "r"(r.w[15]),
          "r"(r.w[16]), "r"(r.w[17]));
}

__device__ __forceinline__ void fs_rl_chain_q123(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%9")
        FS_RL_STEP("%0", "%13", "%14") FS_RL_STEP("%1", "%14", "%15") FS_RL_STEP("%2", "%15", "%16")
        FS_RL_STEP("%3", "%16", "%17") FS_RL_STEP("%4", "%17", "%10") FS_RL_STEP("%5", "%10", "%11")
        FS_RL_STEP("%6", "%11", "%12") FS_RL_STEP("%7", "%12", "%0") FS_RL_STEP("%8", "%0", "%1")
        FS_RL_BORROW_OUT("%9")
        : "+r"(r.w[3]), "+r"(r.w[4]), "+r"(r.w[5]), "+r"(r.w[6]), "+r"(r.w[7]), "+r"(r.w[8]),
          "+r"(r.w[9]), "+r"(r.w[10]), "+r"(r.w[11]), "+r"(r.carry)
        : "r"(r.w[0]), "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[13]), "r"(r.w[14]), "r"(r.w[15]),
          "r"(r.w[16]), "r"(r.w[17]));
}

__device__ __forceinline__ void fs_rl_chain_q234(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%9")
        FS_RL_STEP("%0", "%16", "%17") FS_RL_STEP("%1", "%17", "%10") FS_RL_STEP("%2", "%10", "%11")
        FS_RL_STEP("%3", "%11", "%12") FS_RL_STEP("%4", "%12", "%13") FS_RL_STEP("%5", "%13", "%14")
        FS_RL_STEP("%6", "%14", "%15") FS_RL_STEP("%7", "%15", "%0") FS_RL_STEP("%8", "%0", "%1")
        FS_RL_BORROW_OUT("%9")
        : "+r"(r.w[6]), "+r"(r.w[7]), "+r"(r.w[8]), "+r"(r.w[9]), "+r"(r.w[10]), "+r"(r.w[11]),
          "+r"(r.w[12]), "+r"(r.w[13]), "+r"(r.w[14]), "+r"(r.carry)
        : "r"(r.w[0]), "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[3]), "r"(r.w[4]), "r"(r.w[5]),
          "r"(r.w[16]), "r"(r.w[17]));
}

__device__ __forceinline__ void fs_rl_chain_q345(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%9")
        FS_RL_STEP("%0", "%10", "%11") FS_RL_STEP("%1", "%11", "%12") FS_RL_STEP("%2", "%12", "%13")
        FS_RL_STEP("%3", "%13", "%14") FS_RL_STEP("%4", "%14", "%15") FS_RL_STEP("%5", "%15", "%16")
        FS_RL_STEP("%6", "%16", "%17") FS_RL_STEP("%7", "%17", "%0") FS_RL_STEP("%8", "%0", "%1")
        FS_RL_BORROW_OUT("%9")
        : "+r"(r.w[9]), "+r"(r.w[10]), "+r"(r.w[11]), "+r"(r.w[12]), "+r"(r.w[13]), "+r"(r.w[14]),
          "+r"(r.w[15]), "+r"(r.w[16]), "+r"(r.w[17]), "+r"(r.carry)
        : "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[3]), "r"(r.w[4]), "r"(r.w[5]), "r"(r.w[6]),
          "r"(r.w[7]), "r"(r.w[8]));
}

__device__ __forceinline__ void fs_rl_cycle(FsRanlux &r)
{
    asm(FS_RL_BORROW_IN("%18")
        FS_RL_STEP("%0", "%10", "%11") FS_RL_STEP("%1", "%11", "%12") FS_RL_STEP("%2", "%12", "%13")
        FS_RL_STEP("%3", "%13", "%14") FS_RL_STEP("%4", "%14", "%15") FS_RL_STEP("%5", "%15", "%16")
        FS_RL_STEP("%6", "%16", "%17") FS_RL_STEP("%7", "%17", "%0") FS_RL_STEP("%8", "%0", "%1")
        FS_RL_STEP("%9", "%1", "%2") FS_RL_STEP("%10", "%2", "%3") FS_RL_STEP("%11", "%3", "%4")
        FS_RL_STEP("%12", "%4", "%5") FS_RL_STEP("%13", "%5", "%6") FS_RL_STEP("%14", "%6", "%7")
        FS_RL_STEP("%15", "%7", "%8") FS_RL_STEP("%16", "%8", "%9") FS_RL_STEP("%17", "%9", "%10")
        FS_RL_BORROW_OUT("%18")
        : "+r"(r.w[0]), "+r"(r.w[1]), "+r"(r.w[2]), "+r"(r.w[3]), "+r"(r.w[4]), "+r"(r.w[5]),
          "+r"(r.w[6]), "+r"(r.w[7]), "+r"(r.w[8]), "+r"(r.w[9]), "+r"(r.w[10]), "+r"(r.w[11]),
          "+r"(r.w[12]), "+r"(r.w[13]), "+r"(r.w[14]), "+r"(r.w[15]), "+r"(r.w[16]),
          "+r"(r.w[17]), "+r"(r.carry));
}

// the NQ quads starting at quad Q (the combinations above)
template <int Q, int NQ>
__device__ __forceinline__ void fs_rl_chain(FsRanlux &r)
{
    static_assert(NQ == 1 || (NQ == 2 && (Q == 0 || Q == 4)) || (NQ == 3 && Q <= 3), "no such chain");
    if (NQ == 1 && Q == 0) fs_rl_chain_q0(r);
    if (NQ == 1 && Q == 1) fs_rl_chain_q1(r);
    if (NQ == 1 && Q == 2) fs_rl_chain_q2(r);
    if (NQ == 1 && Q == 3) fs_rl_chain_q3(r);
    if (NQ == 1 && Q == 4) fs_rl_chain_q4(r);
    if (NQ == 1 && Q == 5) fs_rl_chain_q5(r);
    if (NQ == 2 && Q == 0) fs_rl_chain_q01(r);
    if (NQ == 2 && Q == 4) fs_rl_chain_q45(r);
    if (NQ == 3 && Q == 0) fs_rl_chain_q012(r);
    if (NQ == 3 && Q == 1) fs_rl_chain_q123(r);
    if (NQ == 3 && Q == 2) fs_rl_chain_q234(r);
    if (NQ == 3 && Q == 3) fs_rl_chain_q345(r);
}

// digit P of the state, shifted left by 8
template <int P>
__device__ __forceinline__ fs_u32 fs_rl_digit8(const FsRanlux &r)
{
    const int j = P / 4 * 3;
    if (P % 4 == 0) return r.w[j] << 8;
    if (P % 4 == 1) return __funnelshift_l(r.w[j], r.w[j + 1], 16) & 0xFFFFFF00u;
    if (P % 4 == 2) return __funnelshift_l(r.w[j + 1], r.w[j + 2], 24) & 0xFFFFFF00u;
    return r.w[j + 2] & 0xFFFFFF00u;
}

// Generator values leave this part in units of 2^-32 (FS_RL_UNIT): the conversion of a digit
// shifted left by 8, without the multiplication.  A power of two commutes with every rounding
// here (no value is below 2^-48), so a user that multiplies anyway folds it in.
#define FS_RL_UNIT 0x1p-32f

// output of the step that updated digit P (pyopencl-ranluxcl.cl:363-378): a value below 2^-12
// gets the bits of the digit nine steps before, zero becomes 2^-48.  That digit is as it was
// at the step until a skip or the step of its own position in the next cycle.
template <int P>
__device__ __forceinline__ float fs_rl_value(const FsRanlux &r)
{
    const fs_u32 v = fs_rl_digit8<P>(r);
    const float hi = __uint2float_rn(v);
    const float lo = __fmul_rn(__uint2float_rn(fs_rl_digit8<(P + 15) % 24>(r)), 0x1p-24f);
    float out = v < (4096u << 8) ? __fadd_rn(hi, lo) : hi;
    return out == 0.0f ? 0x1p-16f : out;
}

// plain conversions of quad Q, whose chain has run, and the smallest of its digits
template <int Q>
__device__ __forceinline__ fs_u32 fs_rl_plain4(const FsRanlux &r, float *o)
{
    const fs_u32 d0 = fs_rl_digit8<4 * Q>(r), d1 = fs_rl_digit8<4 * Q + 1>(r);
    const fs_u32 d2 = fs_rl_digit8<4 * Q + 2>(r), d3 = fs_rl_digit8<4 * Q + 3>(r);
    o[0] = __uint2float_rn(d0);
    o[1] = __uint2float_rn(d1);
    o[2] = __uint2float_rn(d2);
    o[3] = __uint2float_rn(d3);
    return __vimin3_u32(min(d0, d1), d2, d3);
}

template <int Q>
__device__ __forceinline__ void fs_rl_value4(const FsRanlux &r, float *o)
{
    o[0] = fs_rl_value<4 * Q>(r);
    o[1] = fs_rl_value<4 * Q + 1>(r);
    o[2] = fs_rl_value<4 * Q + 2>(r);
    o[3] = fs_rl_value<4 * Q + 3>(r);
}

// NQ quads starting at quad Q, their steps in one chain: the plain conversions, and the
// small-value correction of fs_rl_value only when some lane of the warp drew a value below 2^-12
// (probability 2^-12 per value).  One vote for all of them, not one a quad: the trimer sweep went
// from 5.53 to 5.21 ms a run, and to 5.11 with the values in units of 2^-32.  The smallest digit in
// three-input minima: 5.00 -> 4.98.
template <int Q, int NQ>
__device__ __forceinline__ void fs_rl_quads(FsRanlux &r, float *o)
{
    fs_rl_chain<Q, NQ>(r);
    fs_u32 least = fs_rl_plain4<Q>(r, o);
    if (NQ > 1) {
        const fs_u32 b = fs_rl_plain4<(Q + 1) % 6>(r, o + 4);
        least = NQ > 2 ? __vimin3_u32(least, b, fs_rl_plain4<(Q + 2) % 6>(r, o + 8)) : min(least, b);
    }
    if (__any_sync(__activemask(), least < (4096u << 8))) {
        fs_rl_value4<Q>(r, o);
        if (NQ > 1) fs_rl_value4<(Q + 1) % 6>(r, o + 4);
        if (NQ > 2) fs_rl_value4<(Q + 2) % 6>(r, o + 8);
    }
}

// NSKIP steps from digit 0, and the frame moved to where they end
template <int NSKIP>
__device__ __forceinline__ void fs_rl_skip(FsRanlux &r)
{
    const int rem = NSKIP % 24, turn = rem / 4 * 3;
#pragma unroll 1
    for (int i = 0; i < NSKIP / 24; i++) fs_rl_cycle(r);
    if (rem > 0) fs_rl_chain_q0(r);
    if (rem > 4) fs_rl_chain_q1(r);
    if (rem > 8) fs_rl_chain_q2(r);
    if (rem > 12) fs_rl_chain_q3(r);
    if (rem > 16) fs_rl_chain_q4(r);
    if (rem > 0) {
        fs_u32 t[18];
#pragma unroll
        for (int j = 0; j < 18; j++) t[j] = r.w[(j + turn) % 18];
#pragma unroll
        for (int j = 0; j < 18; j++) r.w[j] = t[j];
        const fs_u32 p = r.rot + (fs_u32)rem;
        r.rot = p >= 24u ? p - 24u : p;
    }
}

// four outputs (ranluxcl32, in units of 2^-32), then the skip after every 24 outputs
template <int NSKIP>
__device__ __forceinline__ void fs_rl_next4(FsRanlux &r, float &o0, float &o1, float &o2, float &o3)
{
    float o[4];
    switch (r.q) {
    case 0: fs_rl_quads<0, 1>(r, o); break;
    case 1: fs_rl_quads<1, 1>(r, o); break;
    case 2: fs_rl_quads<2, 1>(r, o); break;
    case 3: fs_rl_quads<3, 1>(r, o); break;
    case 4: fs_rl_quads<4, 1>(r, o); break;
    default: fs_rl_quads<5, 1>(r, o); break;
    }
    o0 = o[0]; o1 = o[1]; o2 = o[2]; o3 = o[3];
    if (++r.q == 6u) {
        fs_rl_skip<NSKIP>(r);
        r.q = 0u;
    }
}

// twelve outputs, the same as three calls of next4: straight-line code per starting quad, and
// one copy of the skip (a loop over next4 spends four selects, a branch and eight moves a
// quad; the trimer sweep took 5.96 ms with it and 5.57 ms so, before the single vote)
template <int NSKIP>
__device__ __forceinline__ void fs_rl_next12(FsRanlux &r, float (&c)[12])
{
    const fs_u32 q = r.q;
    if (q < 3u) {
        if (q == 0u) fs_rl_quads<0, 3>(r, c);
        else if (q == 1u) fs_rl_quads<1, 3>(r, c);
        else fs_rl_quads<2, 3>(r, c);
        r.q = q + 3u;
        return;
    }
    if (q == 3u) fs_rl_quads<3, 3>(r, c);
    else if (q == 4u) fs_rl_quads<4, 2>(r, c);
    else fs_rl_quads<5, 1>(r, c);
    fs_rl_skip<NSKIP>(r);
    if (q == 4u) fs_rl_quads<0, 1>(r, c + 8);
    else if (q == 5u) fs_rl_quads<0, 2>(r, c + 4);
    r.q = q - 3u;
}

// ranluxcl_init: three xorshift64 words give eight 24-bit lags, three times; 32 cycles
// of warm-up (pyopencl-ranluxcl.cl:597-725).  Lag a is digit 23 - a.
__device__ __forceinline__ void fs_rl_pack(FsRanlux &r, const fs_u32 (&d)[24])
{
#pragma unroll
    for (int g = 0; g < 6; g++) {
        r.w[3 * g] = d[4 * g] | (d[4 * g + 1] << 24);
        r.w[3 * g + 1] = (d[4 * g + 1] >> 8) | (d[4 * g + 2] << 16);
        r.w[3 * g + 2] = (d[4 * g + 2] >> 16) | (d[4 * g + 3] << 8);
    }
}

__device__ __forceinline__ void fs_rl_seed(FsRanlux &r, fs_u64 x)
{
    fs_u32 d[24];
#pragma unroll
    for (int b = 0; b < 3; b++) {
        fs_u64 w[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            x ^= x << 13;
            x ^= x >> 7;
            x ^= x << 17;
            w[k] = x;
        }
        // 192 bits w0|w1|w2, most significant first, in chunks of 24
        const int a = 23 - 8 * b;
        d[a] = (fs_u32)(w[0] >> 40);
        d[a - 1] = (fs_u32)(w[0] >> 16) & 0xFFFFFFu;
        d[a - 2] = ((fs_u32)(w[0] & 0xFFFFu) << 8) | (fs_u32)(w[1] >> 56);
        d[a - 3] = (fs_u32)(w[1] >> 32) & 0xFFFFFFu;
        d[a - 4] = (fs_u32)(w[1] >> 8) & 0xFFFFFFu;
        d[a - 5] = ((fs_u32)(w[1] & 0xFFu) << 16) | (fs_u32)(w[2] >> 48);
        d[a - 6] = (fs_u32)(w[2] >> 24) & 0xFFFFFFu;
        d[a - 7] = (fs_u32)w[2] & 0xFFFFFFu;
    }
    fs_rl_pack(r, d);
    r.q = 0u;
    r.rot = 0u;
    r.carry = d[0] == 0u ? 0xFFFFFFFFu : 0u;
#pragma unroll 1
    for (int i = 0; i < 32; i++) fs_rl_cycle(r);
}

// Reference table layout <-> packed state.  The table's position (stepnr) is the next step's;
// in24 counts the values since the last skip, except where the skip is a multiple of 24 steps
// (the planar scheme): there it stays untouched and a skip follows the step at position 23.
// A table that a generator has not written (a count or position outside its range) is
// clamped into range.
template <int NSKIP>
__device__ __forceinline__ void fs_rl_load(FsRanlux &r, const fs_u32 *t)
{
    const fs_u32 stepnr = t[27], done = NSKIP % 24 == 0 ? stepnr : t[26];
    r.q = min(done / 4u, 5u);
    r.rot = NSKIP % 24 == 0 ? 0u : (stepnr + 24u - 4u * r.q) % 24u;
    fs_u32 d[24];
#pragma unroll
    for (int f = 0; f < 24; f++) {
        const fs_u32 p = r.rot + (fs_u32)f;
        d[f] = (fs_u32)__fmul_rn(__uint_as_float(t[p < 24u ? 23u - p : 47u - p]), 16777216.0f);
    }
    fs_rl_pack(r, d);
    r.carry = t[24] != 0u ? 0xFFFFFFFFu : 0u;
}

// the words that a generator call changes; word 25 (padding) and, in the planar scheme, word 26
// keep what the table holds
template <int NSKIP>
__device__ __forceinline__ void fs_rl_store(const FsRanlux &r, fs_u32 *t)
{
    fs_u32 d[24];
#pragma unroll
    for (int g = 0; g < 6; g++) {
        d[4 * g] = r.w[3 * g] & 0xFFFFFFu;
        d[4 * g + 1] = __funnelshift_r(r.w[3 * g], r.w[3 * g + 1], 24) & 0xFFFFFFu;
        d[4 * g + 2] = __funnelshift_r(r.w[3 * g + 1], r.w[3 * g + 2], 16) & 0xFFFFFFu;
        d[4 * g + 3] = r.w[3 * g + 2] >> 8;
    }
#pragma unroll
    for (int f = 0; f < 24; f++) {
        const fs_u32 p = r.rot + (fs_u32)f;
        t[p < 24u ? 23u - p : 47u - p] = __float_as_uint(__fmul_rn(__uint2float_rn(d[f]), 0x1p-24f));
    }
    t[24] = r.carry ? __float_as_uint(0x1p-24f) : 0u;
    if (NSKIP % 24 != 0) t[26] = 4u * r.q;
    const fs_u32 p = r.rot + 4u * r.q;
    t[27] = p >= 24u ? p - 24u : p;
}

// a seeded state into a table row that holds nothing yet
template <int NSKIP>
__device__ __forceinline__ void fs_rl_store_new(const FsRanlux &r, fs_u32 *t)
{
    t[25] = 0u;
    t[26] = 0u;
    fs_rl_store<NSKIP>(r, t);
}

// kernel.c:180-190: four buffered values per generator call; the counter starts at 0
// in every launch (kernel.c:557-558)
template <int NSKIP>
struct FsRanluxStream {
    FsRanlux st;
    float b0, b1, b2, b3;  // in units of 2^-32
    fs_u32 count;

    __device__ __forceinline__ float next()
    {
        fs_u32 c = count & 3u;
        if (c == 0u) fs_rl_next4<NSKIP>(st, b0, b1, b2, b3);
        count++;
        return __fmul_rn(c == 0u ? b0 : (c == 1u ? b1 : (c == 2u ? b2 : b3)), FS_RL_UNIT);
    }

    // K consecutive values (K a multiple of 4) in units of 2^-32, the same values next() would
    // return K times: the rem still-buffered values first, then K/4 fresh quadruples, the last rem
    // of which stay buffered.  One branch per K values instead of one per value.
    template <int K>
    __device__ __forceinline__ void next_k(float (&u)[K])
    {
        static_assert(K % 4 == 0, "K must be a multiple of 4");
        const fs_u32 rem = (4u - (count & 3u)) & 3u;
        float c[K];
        if constexpr (K == 12) {
            fs_rl_next12<NSKIP>(st, c);
        } else {
            // one inlined generator call in a rolled loop (the generator is large; K/4 inlined
            // copies cost instruction-cache misses): each quadruple is shifted in at the end
#pragma unroll 1
            for (int q = 0; q < K / 4; q++) {
                float o0, o1, o2, o3;
                fs_rl_next4<NSKIP>(st, o0, o1, o2, o3);
#pragma unroll
                for (int k = 0; k < K - 4; k++) c[k] = c[k + 4];
                c[K - 4] = o0; c[K - 3] = o1; c[K - 2] = o2; c[K - 1] = o3;
            }
        }
        switch (rem) {
        case 0:
#pragma unroll
            for (int k = 0; k < K; k++) u[k] = c[k];
            b0 = c[K - 4]; b1 = c[K - 3]; b2 = c[K - 2]; b3 = c[K - 1];
            break;
        case 1:
            u[0] = b3;
#pragma unroll
            for (int k = 1; k < K; k++) u[k] = c[k - 1];
            b3 = c[K - 1];
            break;
        case 2:
            u[0] = b2; u[1] = b3;
#pragma unroll
            for (int k = 2; k < K; k++) u[k] = c[k - 2];
            b2 = c[K - 2]; b3 = c[K - 1];
            break;
        default:
            u[0] = b1; u[1] = b2; u[2] = b3;
#pragma unroll
            for (int k = 3; k < K; k++) u[k] = c[k - 3];
            b1 = c[K - 3]; b2 = c[K - 2]; b3 = c[K - 1];
            break;
        }
        count += K;
    }
};

// exact FP64 value of an output (zero or a normal number below 1): GB300's FP64 pipe is narrow
__device__ __forceinline__ double fs_rl_f2d(float x)
{
    const fs_u32 u = __float_as_uint(x);
    return __hiloint2double((int)(u ? (u >> 3) + (896u << 20) : 0u), (int)(u << 29));
}

// ranluxcl64 (pyopencl-ranluxcl.cl:893-920) with the same four-value buffering
template <int NSKIP>
struct FsRanluxStream64 {
    FsRanlux st;
    double b0, b1, b2, b3;
    fs_u32 count;

    __device__ __forceinline__ void pair(double &a, double &b)
    {
        float v0, v1, v2, v3;
        fs_rl_next4<NSKIP>(st, v0, v1, v2, v3);
        v0 = __fmul_rn(v0, FS_RL_UNIT);
        v1 = __fmul_rn(v1, FS_RL_UNIT);
        v2 = __fmul_rn(v2, FS_RL_UNIT);
        v3 = __fmul_rn(v3, FS_RL_UNIT);
        if (v0 == 0x1p-48f) v0 = 0.0f;
        if (v2 == 0x1p-48f) v2 = 0.0f;
        // v0 + v1 / 2^24, the exact quotient rounded into the sum: one FP64 operation where a
        // division takes about ten, and the conversions on the integer pipe (five atoms in FP64, 1024
        // walkers, 4 sweeps: 3333 -> 3268 us)
        a = __fma_rn(fs_rl_f2d(v1), 0x1p-24, fs_rl_f2d(v0));
        b = __fma_rn(fs_rl_f2d(v3), 0x1p-24, fs_rl_f2d(v2));
    }

    __device__ __forceinline__ double next()
    {
        fs_u32 c = count & 3u;
        if (c == 0u) {
            pair(b0, b1);
            pair(b2, b3);
        }
        count++;
        return c == 0u ? b0 : (c == 1u ? b1 : (c == 2u ? b2 : b3));
    }
};
