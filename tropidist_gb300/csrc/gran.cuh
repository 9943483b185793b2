// The granule pass: several whole columns (expand, update, select) of the dense sweep in one pass
// over a wide table, every update of the pass applied in registers.
//
// A granule is 4 bytes of the table: 4 entries of uint8, 2 of uint16.  Updates commute, and a run
// of columns with masks h_1, h_2, ... moves a state only along those masks, so the table splits into
// cosets of their span.  A thread owns one coset per step: up to 2^5 granules ("members"), one per
// setting of 5 register dimensions ("slots").  Slot j is the direction of one column's mask, and a
// member's entries are held permuted by the in-granule bits of its directions, so an update is a
// plain pairing of members z and z ^ 2^j at the same register position:
//   N  column that opens and closes no row: min-plus on the pairs of its slot;
//   C  column that closes a row: the slot's two members become one (which of the two is kept is a
//      parity of the other slots and of coset-number bits), the slot is free afterwards;
//   O  column that opens a row: the members double into a free slot (one copy + w): no INF half is
//      read, kept or computed on;
//   A  column that opens a row and closes another: the new row takes the old one's place, w is added
//      where the new row is 1; no slot at all;
//   T  the row of a slot changes places with an in-granule row (a register transposition).
// So a pass of 5 slots takes 7.3 columns of the 31-bit banded plan on average (6 to 8 in its widest
// passes), where a pass that keeps the opened rows' INF halves and the closed rows' dropped halves in its
// registers takes 2 to 3.
//
// A warp's lanes are the lowest coset-number bits, which are the lowest input positions that no
// member direction uses, and the output order keeps the lowest three of them low: a warp reads and
// writes whole 32-byte sectors (usually 128-byte lines) with 4-byte accesses, so the table needs no
// shared-memory staging.
//
// Bound: issue slots (VIADDMNMX, LOP3 and the address arithmetic; 60-68 % of the issue rate on tables of 2^27 to 2^30 entries, the ALU pipe
// next), not HBM: on the 31-bit plan (window 37) a sweep moves 57 GB in 270 passes where the
// chunk-streaming passes moved 181 GB in 735, and takes 19.2 ms instead of 47.2 ms; 26 bits 2.15 instead
// of 4.74 ms; uint16 at 27 bits 1.73 instead of 10.9 ms (tile passes).
#pragma once
#include "tg_common.cuh"

namespace tg {

#define GP_SLOTS 5
#define GP_MEMBERS 32
#define GP_MAXOPS 20
#define GP_MAXK 31           // coset-number bits: 8 by bit, 24 by tables of 4 (the last one spare)

// op codes: a type's slot variants follow each other
// (T: slots 0 and 1 only)
enum GranCode { GC_N = 0, GC_C = 5, GC_O = 10, GC_A = 15, GC_T0 = 16, GC_T1 = 18, GC_I1 = 20, GC_I2 = 21, GC_I3 = 22 };

// A column's weight is paid where a parity over slots, coset-number bits (kmask) and cst is 1 (0 on the
// other copy); d[s] = the weight where the parity includes slot s, else 0.
struct GranOp {
    uint32_t code;
    uint32_t w2;                     // weight in both 16-bit lanes
    uint32_t kmask, cst;
    uint32_t d[5];
    uint32_t lim;                    // pairs (A: members) to go through: the highest dead slots are left out
    uint32_t pad[2];
};

struct GranParams {
    uint64_t ncosets;                // 2^nk
    int nk, nload, nops, pad;        // coset-number bits, slots loaded (0 .. nload - 1)
    uint32_t live_out;               // members stored (bit z)
    uint32_t fin, fout;              // constant parts of the offsets (granules; every offset is 32-bit, so
                                     // tables hold at most 2^GP_MAXBITS granules)
    uint32_t smask0, smask1;         // coset-number bits flipping in-granule bit 0 / 1 of the output
    GranOp ops[GP_MAXOPS];
    uint32_t xin[GP_MEMBERS];        // member z: input offset
    uint2 usel[GP_MEMBERS];          // member z: unpack selectors (even, odd lanes)
    uint2 mout[GP_MEMBERS];          // member z: output offset, pack selector
    uint2 klow[8];                   // (input, output) offsets of coset-number bits 0 .. 7
    uint2 khigh[6][16];              // offsets of bits 8 + 4 g .. 11 + 4 g, by their value
};

template <int EB> struct GranE;
template <> struct GranE<1> { static constexpr int NQ = 2; };    // registers per granule
template <> struct GranE<2> { static constexpr int NQ = 1; };

// The register updates are inline PTX (one VIADDMNMX each): plain intrinsics let the compiler merge the
// tails of the program's cases below, which costs a register move for every operand.
// a = min(a, b + w); uint8 entries sit in 16-bit lanes and cannot wrap
__device__ __forceinline__ void g_addmin(uint32_t &a, uint32_t b, uint32_t w2) {
    asm volatile("{.reg .b32 t;\n\tadd.u16x2 t, %1, %2;\n\tmin.u16x2 %0, t, %0;}" : "+r"(a) : "r"(b), "r"(w2));
}
// a = min(b + w, c)
__device__ __forceinline__ void g_addclamp(uint32_t &a, uint32_t b, uint32_t w2, uint32_t c) {
    asm volatile("{.reg .b32 t;\n\tadd.u16x2 t, %1, %2;\n\tmin.u16x2 %0, t, %3;}" : "=r"(a) : "r"(b), "r"(w2), "r"(c));
}
__device__ __forceinline__ void g_add(uint32_t &a, uint32_t w2) { asm volatile("add.u32 %0, %0, %1;" : "+r"(a) : "r"(w2)); }
__device__ __forceinline__ void g_xor(uint32_t &a, uint32_t b) { asm volatile("xor.b32 %0, %0, %1;" : "+r"(a) : "r"(b)); }
// uint16: b lowered to 65535 - w first, so that b + w saturates at INF
__device__ __forceinline__ uint32_t g_room(uint32_t b, uint32_t w2) { return __vminu2(b, ~w2); }

// a = min(a, b + w), saturating at INF
template <int EB> __device__ __forceinline__ void g_minadd(uint32_t &a, uint32_t b, uint32_t w2) {
    g_addmin(a, EB == 1 ? b : g_room(b, w2), w2);
}
// a = b + w, saturating at INF
template <int EB> __device__ __forceinline__ void g_addsat(uint32_t &a, uint32_t b, uint32_t w2) {
    if (EB == 1) {
        g_addclamp(a, b, w2, 0x00FF00FFu);
    } else {
        a = g_room(b, w2);
        g_add(a, w2);
    }
}
// a = a + w where the result then meets an entry of at most INF in a minimum (uint8: at most 509)
template <int EB> __device__ __forceinline__ void g_addtmp(uint32_t &a, uint32_t w2) {
    if (EB == 2) a = g_room(a, w2);
    g_add(a, w2);
}

__host__ __device__ constexpr int g_ctz(int i) {
    int b = 0;
    while (!((i >> b) & 1)) b++;
    return b;
}
__host__ __device__ constexpr int g_insert0(int i, int s) { return ((i >> s) << (s + 1)) | (i & ((1 << s) - 1)); }

template <int EB, int S> __device__ __forceinline__ void g_op_n(uint32_t (&R)[32 * GranE<EB>::NQ], uint32_t w2,
                                                                uint32_t lim) {
    constexpr int NQ = GranE<EB>::NQ;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        if ((i == 4 || i == 8) && lim <= (uint32_t)i) break;
        const int z = g_insert0(i, S), y = z | (1 << S);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            // the second line may read the new value: min(b, min(a, b + w) + w) = min(b, a + w)
            g_minadd<EB>(R[NQ * z + q], R[NQ * y + q], w2);
            g_minadd<EB>(R[NQ * y + q], R[NQ * z + q], w2);
        }
    }
}

// The members without slot S in Gray order: one slot bit changes between neighbours, so the weight
// of a member (0 or w by the op's parity) follows from the one before by one xor with d[that slot].
template <int EB, int S> __device__ __forceinline__ void g_op_c(uint32_t (&R)[32 * GranE<EB>::NQ], uint32_t w2,
                                                                uint32_t wz, const uint32_t (&d)[5], uint32_t lim) {
    constexpr int NQ = GranE<EB>::NQ;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        if ((i == 4 || i == 8) && lim <= (uint32_t)i) break;
        if (i) { const int b = g_ctz(i); wz ^= d[b < S ? b : b + 1]; }
        const int z = g_insert0(i ^ (i >> 1), S), y = z | (1 << S);
        const uint32_t wo = wz ^ w2;         // parity 0: member z is kept, the other one pays w
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            g_addtmp<EB>(R[NQ * z + q], wz);
            g_minadd<EB>(R[NQ * z + q], R[NQ * y + q], wo);
        }
    }
}

template <int EB, int S> __device__ __forceinline__ void g_op_o(uint32_t (&R)[32 * GranE<EB>::NQ], uint32_t w2,
                                                                uint32_t wz, const uint32_t (&d)[5], uint32_t lim) {
    constexpr int NQ = GranE<EB>::NQ;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        if ((i == 4 || i == 8) && lim <= (uint32_t)i) break;
        if (i) { const int b = g_ctz(i); wz ^= d[b < S ? b : b + 1]; }
        const int z = g_insert0(i ^ (i >> 1), S), y = z | (1 << S);
        const uint32_t wo = wz ^ w2;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            g_addsat<EB>(R[NQ * y + q], R[NQ * z + q], wo);
            g_addsat<EB>(R[NQ * z + q], R[NQ * z + q], wz);
        }
    }
}

template <int EB> __device__ __forceinline__ void g_op_a(uint32_t (&R)[32 * GranE<EB>::NQ], uint32_t wz,
                                                         const uint32_t (&d)[5], uint32_t lim) {
    constexpr int NQ = GranE<EB>::NQ;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        if ((i == 8 || i == 16) && lim <= (uint32_t)i) break;
        if (i) wz ^= d[g_ctz(i)];
        const int z = i ^ (i >> 1);
#pragma unroll
        for (int q = 0; q < NQ; q++) g_addsat<EB>(R[NQ * z + q], R[NQ * z + q], wz);
    }
}

// slot S changes places with in-granule bit 0 of uint8 granules (the register parity)
template <int EB, int S> __device__ __forceinline__ void g_op_t0(uint32_t (&R)[32 * GranE<EB>::NQ]) {
    if constexpr (EB == 1) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int z = g_insert0(i, S), y = z | (1 << S);
            // exchanged by arithmetic: a plain exchange is a renaming, which would tie registers of
            // different members together and cost every case of the program a move per register
            g_xor(R[2 * z + 1], R[2 * y]);
            g_xor(R[2 * y], R[2 * z + 1]);
            g_xor(R[2 * z + 1], R[2 * y]);
        }
    }
}
// ... with the in-granule bit held across the two lanes (bit 1 of uint8 granules, bit 0 of uint16)
template <int EB, int S> __device__ __forceinline__ void g_op_t1(uint32_t (&R)[32 * GranE<EB>::NQ]) {
    constexpr int NQ = GranE<EB>::NQ;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const int z = g_insert0(i, S), y = z | (1 << S);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            // high lane of z with low lane of y; in place, as above
            const uint32_t t = (__byte_perm(R[NQ * z + q], 0u, 0x4432) ^ R[NQ * y + q]) & 0xFFFFu;
            g_xor(R[NQ * y + q], t);
            g_xor(R[NQ * z + q], t << 16);
        }
    }
}

// update whose mask lies inside the granule
template <int EB, int M> __device__ __forceinline__ void g_op_i(uint32_t (&R)[32 * GranE<EB>::NQ], uint32_t w2) {
    constexpr int NQ = GranE<EB>::NQ;
#pragma unroll
    for (int z = 0; z < 32; z++) {
        uint32_t &a = R[z * NQ], &b = R[z * NQ + NQ - 1];
        if (EB == 2) {
            g_minadd<EB>(a, __byte_perm(a, 0u, 0x1032), w2);
        } else if (M == 1) {
            g_minadd<EB>(a, b, w2);
            g_minadd<EB>(b, a, w2);
        } else if (M == 2) {
            g_minadd<EB>(a, __byte_perm(a, 0u, 0x1032), w2);
            g_minadd<EB>(b, __byte_perm(b, 0u, 0x1032), w2);
        } else {
            g_minadd<EB>(a, __byte_perm(b, 0u, 0x1032), w2);
            g_minadd<EB>(b, __byte_perm(a, 0u, 0x1032), w2);
        }
    }
}

template <int EB>
static __device__ __forceinline__ void g_run_ops(const GranParams &P, uint32_t k, uint32_t (&R)[32 * GranE<EB>::NQ]) {
    const int nops = P.nops;
    for (int u = 0; u < nops; u++) {
        const GranOp &O = P.ops[u];
        const uint32_t w2 = O.w2, lim = O.lim;
        const uint32_t wz = ((__popc(k & O.kmask) + O.cst) & 1) ? w2 : 0u;
        const uint32_t d[5] = {O.d[0], O.d[1], O.d[2], O.d[3], O.d[4]};
        switch (O.code) {
            case GC_N + 0: g_op_n<EB, 0>(R, w2, lim); break;
            case GC_N + 1: g_op_n<EB, 1>(R, w2, lim); break;
            case GC_N + 2: g_op_n<EB, 2>(R, w2, lim); break;
            case GC_N + 3: g_op_n<EB, 3>(R, w2, lim); break;
            case GC_N + 4: g_op_n<EB, 4>(R, w2, lim); break;
            case GC_C + 0: g_op_c<EB, 0>(R, w2, wz, d, lim); break;
            case GC_C + 1: g_op_c<EB, 1>(R, w2, wz, d, lim); break;
            case GC_C + 2: g_op_c<EB, 2>(R, w2, wz, d, lim); break;
            case GC_C + 3: g_op_c<EB, 3>(R, w2, wz, d, lim); break;
            case GC_C + 4: g_op_c<EB, 4>(R, w2, wz, d, lim); break;
            case GC_O + 0: g_op_o<EB, 0>(R, w2, wz, d, lim); break;
            case GC_O + 1: g_op_o<EB, 1>(R, w2, wz, d, lim); break;
            case GC_O + 2: g_op_o<EB, 2>(R, w2, wz, d, lim); break;
            case GC_O + 3: g_op_o<EB, 3>(R, w2, wz, d, lim); break;
            case GC_O + 4: g_op_o<EB, 4>(R, w2, wz, d, lim); break;
            case GC_A: g_op_a<EB>(R, wz, d, lim); break;
            case GC_T0 + 0: g_op_t0<EB, 0>(R); break;
            case GC_T0 + 1: g_op_t0<EB, 1>(R); break;
            case GC_T1 + 0: g_op_t1<EB, 0>(R); break;
            case GC_T1 + 1: g_op_t1<EB, 1>(R); break;
            case GC_I1: g_op_i<EB, 1>(R, w2); break;
            case GC_I2: g_op_i<EB, 2>(R, w2); break;
            case GC_I3: g_op_i<EB, 3>(R, w2); break;
            default: break;
        }
    }
}

// Step `step` of a granule pass by one block of 2^TB threads: the cosets step << TB .., one per thread.
// WAIT: a pass launched while the one before it drains waits for that one's table here.
template <int EB, int TB, bool WAIT>
static __device__ __forceinline__ void gran_step(const GranParams &P, uint32_t step, const uint32_t *__restrict__ in,
                                                 uint32_t *__restrict__ out) {
    constexpr int NQ = GranE<EB>::NQ;
    const uint32_t tid = threadIdx.x, k = (step << TB) | tid;
    if ((uint64_t)k >= P.ncosets) return;              // only a pass of fewer cosets than threads
    uint32_t io = P.fin, oo = P.fout;                  // offsets of the thread's coset
#pragma unroll
    for (int b = 0; b < 8; b++)
        if (((b < TB ? tid : k) >> b) & 1u) { io ^= P.klow[b].x; oo ^= P.klow[b].y; }
#pragma unroll
    for (int g = 0; g < 6; g++) {
        const uint2 h = P.khigh[g][(TB <= 8 ? step >> (8 + 4 * g - TB) : k >> (8 + 4 * g)) & 15u];
        io ^= h.x;
        oo ^= h.y;
    }
    const int nload = P.nload;
    if (WAIT) asm volatile("griddepcontrol.wait;" ::: "memory");
    uint32_t R[32 * NQ];                               // members of dead slots hold anything
#pragma unroll
    for (int g = 0; g <= 5; g++) {
        if (g > nload) break;
#pragma unroll
        for (int z = (g ? 1 << (g - 1) : 0); z < (1 << g); z++) R[NQ * z] = __ldcg(in + (io ^ P.xin[z]));
    }
    // parameters in shared memory are read where they are used (as constants they are operands): read ahead
    // they would take the registers that the members need
    asm volatile("" ::: "memory");
#pragma unroll
    for (int g = 0; g <= 5; g++) {
        if (g > nload) break;
#pragma unroll
        for (int z = (g ? 1 << (g - 1) : 0); z < (1 << g); z++) {
            const uint32_t w = R[NQ * z];
            R[NQ * z] = __byte_perm(w, 0u, P.usel[z].x);
            if (EB == 1) R[NQ * z + NQ - 1] = __byte_perm(w, 0u, P.usel[z].y);
        }
    }
    g_run_ops<EB>(P, k, R);
    asm volatile("" ::: "memory");
    // output: in-granule permutation of the member, and of the thread's coset
    uint32_t ts;
    if (EB == 1) ts = ((__popc(k & P.smask0) & 1) ? 0x4444u : 0u) ^ ((__popc(k & P.smask1) & 1) ? 0x2222u : 0u);
    else ts = (__popc(k & P.smask0) & 1) ? 0x2222u : 0u;
    const uint32_t live = P.live_out;
#pragma unroll
    for (int g = 0; g < 8; g++) {
        if (!((live >> (4 * g)) & 15u)) continue;
#pragma unroll
        for (int z = 4 * g; z < 4 * g + 4; z++)
            if ((live >> z) & 1u)
                __stcg(out + (oo ^ P.mout[z].x),
                       __byte_perm(R[NQ * z], EB == 1 ? R[NQ * z + NQ - 1] : 0u, P.mout[z].y ^ ts));
    }
}

}  // namespace tg
