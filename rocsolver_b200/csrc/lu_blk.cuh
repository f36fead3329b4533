// lu_blk.cuh -- right-looking blocked LU (partial pivoting) in separate launches per step.
//
// Replaces the reference's blocked getrf (library/src/lapack/roclapack_getrf.hpp:609-752).
// One step takes a panel of NB = 64 columns of every member:
//   1. lu_panel_kernel       factors the panel (rows j0..m-1), one CTA per member, or a
//                            cluster of CTAs for more than 256 rows;
//   2. lu_swap_trsm_kernel   applies its interchanges to the columns right of it and forms
//                            U12 = L11^{-1} A12;
//   3. lu_gemm_kernel        A22 -= L21 U12 on 64 x 64 tiles of all members;
// and after the last step lu_left_kernel permutes the rows of the finished L columns, all
// later panels' interchanges at once.  Each kernel fills the GPU with its own best shape: the
// panel needs registers and a short serial chain, the update tensor tiles and many CTAs.
// getrf alone, FP64 n = 2048 x 16: 10.8 ms (161 ms with one CTA per member); FP32 n = 501 x 200
// 2.1 ms (2.9).
#pragma once

#include "common.cuh"
#include "lu_cta.cuh" // fma2, WarpTileTF32

namespace rsb {

constexpr int BLK_NB = 64;

// the members of one call
template <typename T>
struct LuBatch
{
    Batch<T> A;
    int m, n, lda;
    int* ipiv;
    int64_t strideP;
    int* info;
    Gate gate;
};

template <typename T>
struct LuMember
{
    T* a;
    int lda, m, n;
    int* piv;
    int* info;
};

template <typename T>
__device__ __forceinline__ bool lu_member(const LuBatch<T>& L, int64_t i, LuMember<T>& M)
{
    if(L.gate.skip(i))
        return false;
    M.a = L.A.at(i);
    M.lda = L.lda;
    M.m = L.m;
    M.n = L.n;
    M.piv = L.ipiv ? L.ipiv + i * L.strideP : nullptr;
    M.info = L.info + i;
    return true;
}

// A panel of this member (one of more than 256 rows, in a cluster) gave up a wait: its factors
// are not valid, its pivots are the identity, and the launches that follow leave it alone.
template <typename T>
__device__ __forceinline__ bool lu_gave_up(const LuBatch<T>& L, const LuMember<T>& M)
{
    return L.m > 256 && *M.info == INT_MIN;
}

// ---------------------------------------------------------------------------- PTX helpers
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;\n" ::
                     : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_rank(const void* p, uint32_t rank)
{
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// 16 bytes to another CTA's shared memory; its mbarrier counts them on arrival
__device__ __forceinline__ void st_async(uint32_t addr, uint4 v, uint32_t mbar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 "
                 "[%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(addr),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init_cluster(uint64_t* b, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n\t"
                 "fence.mbarrier_init.release.cluster;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(b))),
                 "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* b, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(b))),
                 "r"(bytes)
                 : "memory");
}
// stands in for bytes that will not be sent
__device__ __forceinline__ void mbar_complete(uint64_t* b, uint32_t bytes)
{
    asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(b))),
                 "r"(bytes)
                 : "memory");
}
// wait for the phase with this parity; false when it has not come after limit polls of a
// microsecond
constexpr int CLUSTER_WAIT_LIMIT = 1 << 20;
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* b, uint32_t parity, int limit)
{
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(b));
    for(int i = 0; i < limit; ++i)
    {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 1000;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(ok)
                     : "r"(a), "r"(parity)
                     : "memory");
        if(ok)
            return true;
    }
    return false;
}
__device__ __forceinline__ double ld_cluster(uint32_t addr, double)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];\n" : "=d"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr, float)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, int v)
{
    asm volatile("st.shared::cluster.s32 [%0], %1;\n" ::"r"(addr), "r"(v) : "memory");
}
template <int NT>
__device__ __forceinline__ void cta_bar()
{
    asm volatile("bar.sync 1, %0;\n" ::"n"(NT) : "memory");
}
__device__ __forceinline__ void cp_async(double* dst, const double* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async(float* dst, const float* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
template <typename T>
__device__ __forceinline__ void cp_async16(T* dst, const T* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;\n" ::: "memory");
}

// ---------------------------------------------------------------------------- the panel
// One pivot record: the pivot row's entries from the current column to the end of its group
// of 8 columns (shifted: entry 0 is the pivot), the pivot's reciprocal, its key, its position
// (label) and its slot among the CTA's rows.
template <typename T>
struct alignas(16) PanelRec
{
    T row[8];
    T rcp;
    typename KeyOf<T>::type key;
    int label, slot;
};

// upper 32 bits of |x| shifted into the sign's place, plus one: grows with |x|, is never 0,
// and lies below lim for finite x
template <typename T>
struct TopKey;
template <>
struct TopKey<double>
{
    static constexpr uint32_t lim = 0xffe00001u;
    static __device__ __forceinline__ uint32_t of(double x)
    {
        return (uint32_t)__double2hiint(x) * 2u + 1u;
    }
};
template <>
struct TopKey<float>
{
    static constexpr uint32_t lim = 0xff000001u;
    static __device__ __forceinline__ uint32_t of(float x) { return __float_as_uint(x) * 2u + 1u; }
};

template <typename T, int S>
struct PanelShape
{
    static constexpr int RT = 32 * S;           // rows (and row threads) of a CTA
    static constexpr int FW = S > 4 ? S / 4 : 1; // further warps, which factor the column groups
    static constexpr int FS = S / FW;           // rows per lane of those
    static constexpr int NT = RT + 32 * FW;
    static constexpr int LDP = RT + 4;     // conflict-free operand fragments
};
constexpr int PANEL_LDU = BLK_NB + 4;

template <typename T, int NB, int S, bool CL>
struct PanelSmem
{
    T P[NB][PanelShape<T, S>::LDP]; // finished (and the current group's) columns, by row slot
    T R[8][PANEL_LDU];              // the group's pivot rows right of the group, then U
    T U[CL ? 8 : 1][PANEL_LDU];     // (cluster) U of the group; else it takes the place of R
    T L8[8][8];                     // the pivot rows within the group
    PanelRec<T> rec[2][16];         // candidates, double-buffered by column parity; [.][rank, warp]
    PanelRec<T> mine[2];
    uint64_t mbar[2];               // (cluster) arrival of the candidates, by column parity
    int step[32 * S];               // column a row was pivoted at, -1 before
    int label[32 * S];
    int piv[NB];                    // label of each column's pivot row
    int owner[8], slot[8];          // rank and slot of each pivot row of the group
    int mysent[2], sent[16];        // (cluster) columns whose record was sent: own, [rank, warp]
    int failed;                     // (cluster) a wait of this CTA ran out
};

// State of the warp that factors the groups
template <int S>
struct PanelLabels
{
    int lab[S];     // position of each row (row lane + 32 s), -1: no row
    int inf;        // first zero pivot
    uint32_t phase; // (cluster) parity bits of the two barriers
    bool failed;    // (cluster) a wait ran out
};

// Columns c0 .. c0+gb-1 (gb <= 8) of the panel by FW warps: lane i of warp f holds rows i,
// i + 32, ... (S of them, from 32 S f on) of the CTA's rows, 8 entries each, in registers.
// Per column: the rows' keys are reduced in the lane and then by one redux.sync on their
// upper 32 bits, while every lane forms the reciprocal of its own candidate (rows that share
// those bits, infinities and NaN take the full comparison); the winning lane publishes its
// row through shared memory (with two warps the records meet at a barrier of those warps; in
// a cluster every warp sends its candidate to all CTAs, the bytes counted by an mbarrier of
// the receiver); rows are relabelled, not moved; every lane scales and updates its own
// rows.  The column loop is rolled (the update shifts the rows by one entry, so that the
// current column is always entry 0): unrolled, its code did not stay in the instruction
// cache.  A pivot row's remaining entries go to its slot when it is found; what the registers
// of a finished row hold after that is not used.
// A cluster wait that runs out (wait_limit polls) ends the warp's part in the panel: it sends
// and reads no further record, so that the other CTAs' waits run out in turn, and leaves the
// group's rows and slots in range for the threads that go on to the barriers.
// Time of one 64-column FP64 panel alone on an SM: 64 rows (S = 2) 36 us, 128 rows 33 us; 256
// rows took 58 us with one warp of 8 rows a lane, which is why they have two.
template <typename T, int NB, int SC, bool PIVOT, bool CL>
__device__ __forceinline__ void panel_group(PanelSmem<T, NB, SC, CL>& sm,
                                            PanelLabels<PanelShape<T, SC>::FS>& st, int f, int c0,
                                            int gb, int j0, int rank, int nrank, int wait_limit)
{
    constexpr int S = PanelShape<T, SC>::FS, FW = PanelShape<T, SC>::FW;
    using K = typename KeyOf<T>::type;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int(&lab)[S] = st.lab;
    T x[S][8];
#pragma unroll
    for(int s = 0; s < S; ++s)
#pragma unroll
        for(int k = 0; k < 8; ++k)
            x[s][k] = sm.P[c0 + k][f * 32 * S + lane + 32 * s];
    int k = 0;
#pragma unroll 1
    for(; k < gb; ++k)
    {
        if(CL && st.failed)
            break;
        const int c = c0 + k;
        // (selections, no branches: a divergent branch per row costs more than the row)
        uint32_t hv[S];
        T xv[S];
        int sv[S];
#pragma unroll
        for(int s = 0; s < S; ++s)
        {
            const bool act = PIVOT ? lab[s] >= c : lab[s] == c;
            hv[s] = act ? TopKey<T>::of(x[s][0]) : 0u;
            xv[s] = x[s][0];
            sv[s] = s;
        }
#pragma unroll
        for(int d = 1; d < S; d *= 2)
#pragma unroll
            for(int s = 0; s < S; s += 2 * d)
            {
                const bool up = hv[s + d] > hv[s];
                hv[s] = up ? hv[s + d] : hv[s];
                xv[s] = up ? xv[s + d] : xv[s];
                sv[s] = up ? sv[s + d] : sv[s];
            }
        const uint32_t best = hv[0];
        T bx = xv[0];
        int bs = sv[0];
        const uint32_t top = __reduce_max_sync(full, best);
        T brcp = Lim<T>::rcp(bx);
        bool win = best == top;
        unsigned equal = 0;
#pragma unroll
        for(int s = 0; s < S; ++s)
            equal += (PIVOT ? lab[s] >= c : lab[s] == c) && TopKey<T>::of(x[s][0]) == top ? 1u : 0u;
        if(__reduce_add_sync(full, equal) != 1u || top >= TopKey<T>::lim)
        {
            // the full key, then the smallest label (LAPACK: first index of the maximum)
            K bk = 0;
            int bl = INT_MAX;
#pragma unroll
            for(int s = 0; s < S; ++s)
            {
                const bool act = PIVOT ? lab[s] >= c : lab[s] == c;
                const K key = pivot_key(x[s][0], lab[s] == c);
                const bool up = act && (bl == INT_MAX || key > bk || (key == bk && lab[s] < bl));
                bk = up ? key : bk;
                bl = up ? lab[s] : bl;
                bx = up ? x[s][0] : bx;
                bs = up ? s : bs;
            }
            K gk;
            const int wl = warp_argmax(bk, bl, bl != INT_MAX, &gk);
            win = bl == wl && bl != INT_MAX;
            brcp = Lim<T>::rcp(bx);
        }
        PanelRec<T>& out = CL ? sm.mine[f] : sm.rec[k & 1][f];
        if((CL || FW > 1) && top == 0 && lane == 0)
            out.label = INT_MAX; // no row of this warp takes part
        if(win && top != 0)
        {
            switch(bs)
            {
#define RSB_PUBLISH(Q)                                                                         \
    case Q:                                                                                    \
        if constexpr(Q < S)                                                                    \
        {                                                                                      \
            _Pragma("unroll") for(int j = 0; j < 8; ++j) out.row[j] = x[Q < S ? Q : 0][j];     \
            out.label = lab[Q < S ? Q : 0];                                                    \
            if(CL || FW > 1)                                                                   \
                out.key = pivot_key(bx, lab[Q < S ? Q : 0] == c);                              \
        }                                                                                      \
        break;
                RSB_PUBLISH(0)
                RSB_PUBLISH(1)
                RSB_PUBLISH(2)
                RSB_PUBLISH(3)
#undef RSB_PUBLISH
            }
            out.rcp = brcp;
            out.slot = f * 32 * S + lane + 32 * bs;
        }
        __syncwarp();
        int w = 0;
        if(CL)
        {
            constexpr int CH = sizeof(PanelRec<T>) / 16;
            const int nrec = nrank * FW;
            if(lane == 0 && f == 0)
                mbar_expect(&sm.mbar[k & 1], (uint32_t)(nrec * sizeof(PanelRec<T>)));
            for(int e = lane; e < nrank * CH; e += 32)
            {
                const int to = e / CH, q = e % CH;
                st_async(map_rank(&sm.rec[k & 1][rank * FW + f], to) + 16 * q,
                         reinterpret_cast<const uint4*>(&sm.mine[f])[q],
                         map_rank(&sm.mbar[k & 1], to));
            }
            const bool came =
                mbar_wait_cluster(&sm.mbar[k & 1], (st.phase >> (k & 1)) & 1u, wait_limit);
            st.failed = !__all_sync(full, came);
            if(st.failed)
            {
                // the records of this column may be unwritten
                if(lane == 0)
                    sm.mysent[f] = c + 1;
                break;
            }
            st.phase ^= 1u << (k & 1);
            const PanelRec<T>& rl = sm.rec[k & 1][lane & 15];
            const bool in = lane < nrec && rl.label != INT_MAX;
            const int lb = in ? rl.label : INT_MAX;
            K gk;
            const int gl = warp_argmax(in ? rl.key : K(0), lb, in, &gk);
            w = max(0, __ffs(__ballot_sync(full, in && lb == gl)) - 1);
        }
        else if constexpr(FW > 1)
        {
            asm volatile("bar.sync 2, %0;\n" ::"n"(32 * FW) : "memory");
            const PanelRec<T>&r0 = sm.rec[k & 1][0], &r1 = sm.rec[k & 1][1];
            const int l0 = r0.label, l1 = r1.label;
            const K k0 = r0.key, k1 = r1.key;
            w = l1 != INT_MAX && (l0 == INT_MAX || k1 > k0 || (k1 == k0 && l1 < l0)) ? 1 : 0;
        }
        const PanelRec<T>& rc = sm.rec[k & 1][w];
        const int wl = rc.label, wslot = rc.slot & (32 * SC - 1);
        w = CL ? w / FW : 0; // rank that holds the pivot row
        const T r = rc.rcp;
        T rw[8];
#pragma unroll
        for(int j = 0; j < 8; ++j)
            rw[j] = rc.row[j];
        const T p = rw[0];
        // LAPACK getf2 scaling: reciprocal when |pivot| >= sfmin, else division; a zero pivot
        // leaves the column unscaled
        if(fabs(p) >= Lim<T>::sfmin())
        {
#pragma unroll
            for(int s = 0; s < S; ++s)
                x[s][0] *= r;
        }
        else if(p != T(0))
        {
#pragma unroll
            for(int s = 0; s < S; ++s)
                x[s][0] = x[s][0] / p;
        }
        else if(st.inf == 0)
            st.inf = j0 + c + 1;
#pragma unroll
        for(int s = 0; s < S; ++s)
        {
            lab[s] = lab[s] == wl ? c : (lab[s] == c ? wl : lab[s]);
            const T l = x[s][0];
            if(lab[s] > c)
                sm.P[c][f * 32 * S + lane + 32 * s] = l;
#pragma unroll
            for(int j = 1; j < 4; ++j)
                x[s][j - 1] = fma(-l, rw[j], x[s][j]);
            x[s][3] = fma(-l, rw[4], x[s][4]);
            if(k < 3) // columns 5.. of the shifted row are still inside the group
            {
#pragma unroll
                for(int j = 5; j < 8; ++j)
                    x[s][j - 1] = fma(-l, rw[j], x[s][j]);
            }
        }
        // off the serial path: the pivot row's remaining entries, the pivot
        if(lane == 0 && f == 0)
        {
            if(w == rank)
            {
                sm.step[wslot] = c;
#pragma unroll
                for(int j = 0; j < 8; ++j)
                    if(j < gb - k)
                        sm.P[c + j][wslot] = rw[j];
            }
            sm.owner[k] = w;
            sm.slot[k] = wslot;
            sm.piv[c] = wl;
        }
    }
    if(CL && st.failed && f == 0 && lane < 8)
    {
        if(lane >= k)
        {
            sm.owner[lane] = rank;
            sm.slot[lane] = 0;
            sm.piv[c0 + lane] = c0 + lane;
        }
    }
    // the pivot rows' multipliers within the group, for U of the columns right of it
    if constexpr(FW > 1)
        asm volatile("bar.sync 2, %0;\n" ::"n"(32 * FW) : "memory");
    else
        __syncwarp();
    if(gb == 8 && f == 0)
    {
#pragma unroll
        for(int e = lane; e < 64; e += 32)
        {
            const int i = e >> 3, k = e & 7;
            if(k < i && sm.owner[i] == rank)
                sm.L8[i][k] = sm.P[c0 + k][sm.slot[i]];
        }
    }
}

// v[ch - 1] = v[ch] - A U for the chunks lo <= ch < hi (ch - 1 = -1: d).  A is the group's
// multipliers of this lane's rows (P at the group's first column and the lane's first row), U
// starts at the chunks' first column.  FP64: tensor products, the A fragments kept (a).
template <typename T, int NB>
struct PanelUpdate;

template <int NB>
struct PanelUpdate<double, NB>
{
    static constexpr int NC = NB / 8 - 1;
    double a[2][4]; // k = 4 h + q
    __device__ __forceinline__ void load(const double* P, int ldp)
    {
        const int q = threadIdx.x & 3;
#pragma unroll
        for(int h = 0; h < 2; ++h)
#pragma unroll
            for(int i = 0; i < 4; ++i)
                a[h][i] = -P[(4 * h + q) * ldp + 8 * i];
    }
    __device__ __forceinline__ void chunk(double (&d)[4][2], const double (&c)[4][2],
                                          const double* U) const
    {
        const int g = (threadIdx.x >> 2) & 7, q = threadIdx.x & 3;
        double t[4][2];
        const double b0 = U[q * PANEL_LDU + g], b1 = U[(4 + q) * PANEL_LDU + g];
#pragma unroll
        for(int i = 0; i < 4; ++i)
            asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                         "{%0, %1}, {%2}, {%3}, {%4, %5};\n"
                         : "=d"(t[i][0]), "=d"(t[i][1])
                         : "d"(a[0][i]), "d"(b0), "d"(c[i][0]), "d"(c[i][1]));
#pragma unroll
        for(int i = 0; i < 4; ++i)
            asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                         "{%0, %1}, {%2}, {%3}, {%4, %5};\n"
                         : "=d"(d[i][0]), "=d"(d[i][1])
                         : "d"(a[1][i]), "d"(b1), "d"(t[i][0]), "d"(t[i][1]));
    }
    __device__ __forceinline__ void first(double (&d)[4][2], double (&v)[NC][4][2],
                                          const double* U, const double*, int) const
    {
        chunk(d, v[0], U);
    }
    __device__ __forceinline__ void others(double (&v)[NC][4][2], const double* U, const double*,
                                           int, int hi) const
    {
#pragma unroll
        for(int ch = 1; ch < NC; ++ch)
        {
            if(ch >= hi)
                break;
            chunk(v[ch - 1], v[ch], U + 8 * ch);
        }
    }
};

template <int NB>
struct PanelUpdate<float, NB>
{
    static constexpr int NC = NB / 8 - 1;
    __device__ __forceinline__ void load(const float*, int) {}
    __device__ __forceinline__ void first(float (&d)[4][2], float (&v)[NC][4][2], const float* U,
                                          const float* P, int ldp) const
    {
        const int q = threadIdx.x & 3;
        float2 t[4];
#pragma unroll
        for(int i = 0; i < 4; ++i)
            t[i] = make_float2(v[0][i][0], v[0][i][1]);
#pragma unroll
        for(int k = 0; k < 8; ++k)
        {
            const float2 u = *reinterpret_cast<const float2*>(U + k * PANEL_LDU + 2 * q);
#pragma unroll
            for(int i = 0; i < 4; ++i)
                fma2(t[i], -P[k * ldp + 8 * i], u.x, u.y);
        }
#pragma unroll
        for(int i = 0; i < 4; ++i)
        {
            d[i][0] = t[i].x;
            d[i][1] = t[i].y;
        }
    }
    __device__ __forceinline__ void others(float (&v)[NC][4][2], const float* U, const float* P,
                                           int ldp, int hi) const
    {
        const int q = threadIdx.x & 3;
#pragma unroll
        for(int ch = 1; ch < NC; ++ch)
#pragma unroll
            for(int i = 0; i < 4; ++i)
#pragma unroll
                for(int e = 0; e < 2; ++e)
                    v[ch - 1][i][e] = v[ch][i][e];
#pragma unroll 2
        for(int k = 0; k < 8; ++k)
        {
            float a[4];
#pragma unroll
            for(int i = 0; i < 4; ++i)
                a[i] = -P[k * ldp + 8 * i];
#pragma unroll
            for(int ch = 1; ch < NC; ++ch)
            {
                if(ch >= hi)
                    break;
                const float2 u = *reinterpret_cast<const float2*>(U + k * PANEL_LDU + 8 * ch + 2 * q);
#pragma unroll
                for(int i = 0; i < 4; ++i)
                {
                    float2 t = make_float2(v[ch - 1][i][0], v[ch - 1][i][1]);
                    fma2(t, a[i], u.x, u.y);
                    v[ch - 1][i][0] = t.x;
                    v[ch - 1][i][1] = t.y;
                }
            }
        }
    }
};

// The panel at (j0, j0): rows j0..m-1 (at most 32 S a CTA), jb = min(NB, min(m, n) - j0) columns.  The row warps
// hold the columns right of the current group of 8 in registers, in tensor-accumulator
// layout; the group itself is factored by one warp, or two for 256 rows, from shared memory
// (panel_group).  Then
// the group's pivot rows are published, U of the group is formed (one thread per column, 8 x
// 8 unit-lower substitution) and the rows take the rank-8 update: first the next group's
// columns, which go to shared memory, then, while that group is being factored, the
// others.  The update moves chunk ch to register chunk ch - 1, so that the group loop is one
// copy of the code.
// CL: a cluster of CTAs, each with 32 * S of the rows; candidates and pivot rows cross it
// through distributed shared memory.
template <typename T, int NB, int S, bool PIVOT, bool CL>
__global__ void __launch_bounds__(PanelShape<T, S>::NT,
                                  S <= 2   ? (sizeof(T) == 8 ? 4 : 6)
                                  : S <= 4 ? (sizeof(T) == 8 ? 2 : 3)
                                           : (sizeof(T) == 8 || CL ? 1 : 2))
    lu_panel_kernel(LuBatch<T> L, int j0, int wait_limit)
{
    using SH = PanelShape<T, S>;
    constexpr int RT = SH::RT, NT = SH::NT, NC = NB / 8 - 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Smem = PanelSmem<T, NB, S, CL>;
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    int nrank = 1, rank = 0;
    if(CL)
    {
        asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(nrank));
        rank = cluster_rank();
    }
    LuMember<T> M;
    if(!lu_member(L, blockIdx.x / nrank, M) || (j0 > 0 && lu_gave_up(L, M)))
        return;
    const int mn = min(M.m, M.n), mp = M.m - j0;
    const int jb = min(NB, mn - j0);
    const int rbase = rank * RT; // this CTA's rows of the panel
    const int mc = max(0, min(RT, mp - rbase));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ngroup = (jb + 7) / 8;
    if(CL)
    {
        if(tid == 0)
        {
            mbar_init_cluster(&sm.mbar[0], 1);
            mbar_init_cluster(&sm.mbar[1], 1);
            sm.failed = 0;
            sm.mysent[0] = sm.mysent[1] = jb;
        }
        cluster_sync_all(); // every CTA's barriers are ready before a candidate is sent
    }
    constexpr int FS = SH::FS;
    const int f = warp - S; // factoring warp's number
    PanelLabels<FS> lb;
    lb.inf = 0;
    lb.phase = 0;
    lb.failed = false;
#pragma unroll
    for(int s = 0; s < FS; ++s)
    {
        const int row = f * 32 * FS + lane + 32 * s;
        lb.lab[s] = row < mc ? rbase + row : -1;
    }

    auto rows = [&]() {
        const int g = lane >> 2, q = lane & 3;
        const int r0 = warp * 32 + g; // this lane's rows: r0 + 8 i
        T v[NC][4][2];
#pragma unroll
        for(int ch = 0; ch <= NC; ++ch)
#pragma unroll
            for(int e = 0; e < 2; ++e)
#pragma unroll
                for(int i = 0; i < 4; ++i)
                {
                    const int r = r0 + 8 * i, c = 8 * ch + 2 * q + e;
                    const T t = (r < mc && c < jb)
                                    ? RSB_AT(M.a, j0 + rbase + r, j0 + c, M.lda, M.m, M.n)
                                    : T(0);
                    if(ch == 0)
                        sm.P[c][r] = t;
                    else
                        v[ch > 0 ? ch - 1 : 0][i][e] = t;
                }
        sm.step[tid] = -1;
        PanelUpdate<T, NB> up;
#pragma unroll 1
        for(int gi = 0; gi < ngroup; ++gi)
        {
            const int c0 = 8 * gi, rest = ngroup - gi - 1; // chunks right of the group
            const T* U = CL ? &sm.U[0][0] : &sm.R[0][0];
            cta_bar<NT>();
            if(gi > 0)
            {
                // the rest of the previous group's update, beside the factorisation
                up.others(v, U, &sm.P[c0 - 8][r0], SH::LDP, rest + 1);
            }
            cta_bar<NT>();
            if(rest > 0)
            {
                int st[4];
#pragma unroll
                for(int i = 0; i < 4; ++i)
                {
                    st[i] = sm.step[r0 + 8 * i];
                    if(st[i] >= c0)
                    {
#pragma unroll
                        for(int ch = 0; ch < NC; ++ch)
                        {
                            sm.R[st[i] - c0][8 * ch + 2 * q] = v[ch][i][0];
                            sm.R[st[i] - c0][8 * ch + 2 * q + 1] = v[ch][i][1];
                        }
                    }
                }
                if(CL)
                    cluster_sync_all();
                else
                    cta_bar<NT>();
                if(tid < 8 * rest)
                {
                    T r[8];
#pragma unroll
                    for(int k = 0; k < 8; ++k)
                        r[k] = CL ? ld_cluster(map_rank(&sm.R[k][tid], sm.owner[k]), T(0))
                                  : sm.R[k][tid];
#pragma unroll
                    for(int k = 0; k < 8; ++k)
#pragma unroll
                        for(int i = k + 1; i < 8; ++i)
                            r[i] = fma(-(CL ? ld_cluster(map_rank(&sm.L8[i][k], sm.owner[i]), T(0))
                                            : sm.L8[i][k]),
                                       r[k], r[i]);
#pragma unroll
                    for(int k = 0; k < 8; ++k)
                    {
                        (CL ? sm.U : sm.R)[k][tid] = r[k];
                        if(!CL || sm.owner[k] == rank) // the finished row's columns
                            sm.P[c0 + 8 + tid][sm.slot[k]] = r[k];
                    }
                }
                cta_bar<NT>();
                up.load(&sm.P[c0][r0], SH::LDP);
                T d[4][2];
                up.first(d, v, U, &sm.P[c0][r0], SH::LDP);
#pragma unroll
                for(int i = 0; i < 4; ++i)
                    if(st[i] < 0)
                    {
                        sm.P[c0 + 8 + 2 * q][r0 + 8 * i] = d[i][0];
                        sm.P[c0 + 9 + 2 * q][r0 + 8 * i] = d[i][1];
                    }
            }
        }
    };

    if(warp >= S)
    {
#pragma unroll 1
        for(int gi = 0; gi < ngroup; ++gi)
        {
            cta_bar<NT>();
            panel_group<T, NB, S, PIVOT, CL>(sm, lb, f, 8 * gi, min(8, jb - 8 * gi), j0, rank,
                                              nrank, wait_limit);
            cta_bar<NT>();
            if(gi + 1 < ngroup)
            {
                if(CL)
                    cluster_sync_all();
                else
                    cta_bar<NT>();
                cta_bar<NT>();
            }
        }
    }
    else
        rows();
    if(warp >= S)
    {
#pragma unroll
        for(int s = 0; s < FS; ++s)
            sm.label[f * 32 * FS + lane + 32 * s] = lb.lab[s];
        if(PIVOT && rank == 0 && f == 0)
        {
            __syncwarp();
            for(int c = lane; c < jb; c += 32)
                M.piv[j0 + c] = j0 + sm.piv[c] + 1;
        }
        if(lane == 0 && rank == 0 && f == 0 && (j0 == 0 || (lb.inf != 0 && *M.info == 0)))
            *M.info = lb.inf;
        if(CL)
        {
            if(lane == 0 && lb.failed)
                sm.failed = 1;
            if(lane < nrank)
                st_cluster(map_rank(&sm.sent[rank * SH::FW + f], lane), sm.mysent[f]);
        }
    }
    cta_bar<NT>();
    // finished columns to their final positions (all of the panel was read at the start)
    if(tid < mc && !(CL && sm.failed))
    {
        const int pos = sm.label[tid];
#pragma unroll 8
        for(int k = 0; k < jb; ++k)
            RSB_AT(M.a, j0 + pos, j0 + k, M.lda, M.m, M.n) = sm.P[k][tid];
    }
    if(CL)
    {
        cluster_sync_all(); // no CTA leaves while its shared memory may be read
        if(sm.failed)
        {
            // rank 0's pivots and info are written: identity pivots and INT_MIN over them
            for(int c = j0 + tid; PIVOT && c < mn; c += NT)
                M.piv[c] = c + 1;
            if(tid == 0)
                *M.info = INT_MIN;
            // ... nor while a record is on its way to it.  Factoring warp 0 expected mysent[0]
            // columns; of the last of them and the next, wait for the records that were sent.
            if(warp == S && lane == 0 && lb.failed)
            {
                constexpr uint32_t RB = sizeof(PanelRec<T>);
                const int nrec = nrank * SH::FW, last = sm.mysent[0] - 1;
                int n0 = 0, n1 = 0;
                for(int i = 0; i < nrec; ++i)
                {
                    n0 += sm.sent[i] > last;
                    n1 += sm.sent[i] > last + 1;
                }
                if(n0 < nrec)
                    mbar_complete(&sm.mbar[last & 1], (nrec - n0) * RB);
                mbar_wait_cluster(&sm.mbar[last & 1], (lb.phase >> (last & 1)) & 1u,
                                  CLUSTER_WAIT_LIMIT);
                if(n1 > 0)
                {
                    mbar_expect(&sm.mbar[(last + 1) & 1], n1 * RB);
                    mbar_wait_cluster(&sm.mbar[(last + 1) & 1],
                                      (lb.phase >> ((last + 1) & 1)) & 1u, CLUSTER_WAIT_LIMIT);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------- U12
// The interchanges of the panel at j0 on 64 columns right of it, then U12 = L11^{-1} A12 for
// them.  A row of the panel's top jb positions may come from anywhere; a position below them
// either keeps its row or takes one of the original top rows.  cp.async gathers L11 and the
// sources of the top positions (all loads in flight at once); then the displaced top rows are
// copied down, whole columns by one warp.  The substitution takes blocks of 16 rows: the
// finished rows' part (FP64: tensor tiles, one warp per 16 columns; FP32: in the column's
// thread), then 16 x 16 unit-lower substitution with one thread per column.  Bound by the gather
// (FP64 n = 1024 x 40: 15 launches 0.79 ms, 1.86 GB of DRAM traffic).
constexpr int TRSM_NT = 128, TRSM_CW = 64;

template <typename T>
struct TrsmSmem
{
    T L[BLK_NB][BLK_NB + 4];   // [k][i] = L11(i, k); only i > k is used
    T X[TRSM_CW][BLK_NB + 1];  // [col][k]
    int piv[BLK_NB], src[BLK_NB], dst[BLK_NB];
};

// rows ib..ib+15 of 16 columns -= L(ib.., 0..ib-1) X as a 16 x 16 tensor tile of one warp;
// L [k][i], x [column][k]
__device__ __forceinline__ void trsm_tile(const double (*L)[BLK_NB + 4], double* x, int ib)
{
    constexpr int LD = BLK_NB + 1;
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    double acc[2][2][2];
#pragma unroll
    for(int i = 0; i < 2; ++i)
#pragma unroll
        for(int j = 0; j < 2; ++j)
#pragma unroll
            for(int e = 0; e < 2; ++e)
                acc[i][j][e] = x[(8 * j + 2 * q + e) * LD + ib + 8 * i + g];
#pragma unroll 4
    for(int k = 0; k < ib; k += 4)
    {
        double a[2], b[2];
#pragma unroll
        for(int i = 0; i < 2; ++i)
        {
            a[i] = -L[k + q][ib + 8 * i + g];
            b[i] = x[(8 * i + g) * LD + k + q];
        }
#pragma unroll
        for(int i = 0; i < 2; ++i)
#pragma unroll
            for(int j = 0; j < 2; ++j)
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                             "{%0, %1}, {%2}, {%3}, {%0, %1};\n"
                             : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
                             : "d"(a[i]), "d"(b[j]));
    }
#pragma unroll
    for(int i = 0; i < 2; ++i)
#pragma unroll
        for(int j = 0; j < 2; ++j)
#pragma unroll
            for(int e = 0; e < 2; ++e)
                x[(8 * j + 2 * q + e) * LD + ib + 8 * i + g] = acc[i][j][e];
}

template <typename T, bool PIVOT>
__global__ void __launch_bounds__(TRSM_NT, sizeof(T) == 8 ? 3 : 5)
    lu_swap_trsm_kernel(LuBatch<T> L, int j0, int chunks)
{
    constexpr int NB = BLK_NB, NT = TRSM_NT, CW = TRSM_CW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TrsmSmem<T>& sm = *reinterpret_cast<TrsmSmem<T>*>(smem_raw);
    LuMember<T> M;
    if(!lu_member(L, blockIdx.x / chunks, M) || lu_gave_up(L, M))
        return;
    const int jb = min(NB, min(M.m, M.n) - j0);
    const int cfirst = j0 + jb + (blockIdx.x % chunks) * CW;
    const int ncol = min(CW, M.n - cfirst);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for(int e = tid; e < NB * NB; e += NT)
    {
        const int i = e & (NB - 1), k = e / NB;
        if(i < jb && k < jb && i > k)
            cp_async(&sm.L[k][i], &RSB_AT(M.a, j0 + i, j0 + k, M.lda, M.m, M.n));
    }
    if(PIVOT)
    {
        if(tid < jb)
        {
            RSB_CHECK_PIV(M.piv[j0 + tid], M.m, __LINE__);
            sm.piv[tid] = M.piv[j0 + tid] - 1 - j0;
        }
        __syncthreads();
        int x = tid & (NB - 1);
        if(tid < NB)
        {
#pragma unroll 8
            for(int k = jb - 1; k >= 0; --k)
            {
                const int p = sm.piv[k];
                x = x == k ? p : (x == p ? k : x);
            }
            sm.src[tid] = x; // position tid receives row x
        }
        else
        {
#pragma unroll 8
            for(int k = 0; k < jb; ++k)
            {
                const int p = sm.piv[k];
                x = x == k ? p : (x == p ? k : x);
            }
            sm.dst[tid - NB] = x; // row tid - NB goes to position x
        }
        __syncthreads();
    }
    int src[2], dst[2];
#pragma unroll
    for(int h = 0; h < 2; ++h)
    {
        src[h] = PIVOT ? sm.src[lane + 32 * h] : lane + 32 * h;
        dst[h] = PIVOT ? sm.dst[lane + 32 * h] : -1;
    }
    for(int c = warp; c < ncol; c += NT / 32)
#pragma unroll
        for(int h = 0; h < 2; ++h)
        {
            const int i = lane + 32 * h;
            if(i < jb)
                cp_async(&sm.X[c][i], &RSB_AT(M.a, j0 + src[h], cfirst + c, M.lda, M.m, M.n));
        }
    cp_async_wait();
    __syncthreads();
    if(PIVOT)
        for(int c0 = warp * 16; c0 < ncol; c0 += NT / 2)
        {
            // every source of these columns has been read
            T d[8][2];
#pragma unroll
            for(int u0 = 0; u0 < 16; u0 += 8)
            {
#pragma unroll
                for(int u = 0; u < 8; ++u)
#pragma unroll
                    for(int h = 0; h < 2; ++h)
                        if(c0 + u0 + u < ncol && lane + 32 * h < jb && dst[h] >= jb)
                            d[u][h] = RSB_AT(M.a, j0 + lane + 32 * h, cfirst + c0 + u0 + u, M.lda,
                                             M.m, M.n);
#pragma unroll
                for(int u = 0; u < 8; ++u)
#pragma unroll
                    for(int h = 0; h < 2; ++h)
                        if(c0 + u0 + u < ncol && lane + 32 * h < jb && dst[h] >= jb)
                            RSB_AT(M.a, j0 + dst[h], cfirst + c0 + u0 + u, M.lda, M.m, M.n) =
                                d[u][h];
            }
        }
#pragma unroll 1
    for(int ib = 0; ib < jb; ib += 16)
    {
        if constexpr(sizeof(T) == 8)
        {
            if(ib > 0 && warp * 16 < ncol)
                trsm_tile(sm.L, &sm.X[warp * 16][0], ib);
            __syncthreads();
        }
        if(tid < ncol)
        {
            T acc[16];
            T* x = sm.X[tid];
#pragma unroll
            for(int r = 0; r < 16; ++r)
                acc[r] = x[ib + r];
            if constexpr(sizeof(T) == 4)
            {
#pragma unroll 2
                for(int k = 0; k < ib; ++k)
                {
                    const T xk = x[k];
#pragma unroll
                    for(int r = 0; r < 16; ++r)
                        acc[r] = fma(-sm.L[k][ib + r], xk, acc[r]);
                }
            }
#pragma unroll
            for(int r = 0; r < 16; ++r)
#pragma unroll
                for(int q = r + 1; q < 16; ++q)
                    acc[q] = fma(-sm.L[ib + r][ib + q], acc[r], acc[q]);
#pragma unroll
            for(int r = 0; r < 16; ++r)
                x[ib + r] = acc[r];
        }
        if constexpr(sizeof(T) == 8)
            __syncthreads();
    }
    __syncthreads();
    for(int c = warp; c < ncol; c += NT / 32)
#pragma unroll
        for(int h = 0; h < 2; ++h)
        {
            const int i = lane + 32 * h;
            if(i < jb)
                RSB_AT(M.a, j0 + i, cfirst + c, M.lda, M.m, M.n) = sm.X[c][i];
        }
}

// ---------------------------------------------------------------------------- A22
// Warp tiles of 32 x 32 on operands sA[k][row] and sB ([col][k] for B_BY_COL, else [k][col]).
constexpr int GEMM_LD = 68; // = 4 mod 32 (32-bit) and 4 mod 16 (64-bit): no bank conflicts

template <typename T, bool TC>
struct GemmTile;

template <>
struct GemmTile<double, false>
{
    double acc[4][4][2];
    static constexpr bool B_BY_COL = true;
    template <bool BY_COL = true>
    __device__ __forceinline__ void mma(const double* sA, const double* sB, int r0, int c0, int kk)
    {
        const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll 2
        for(int k0 = 0; k0 < kk; k0 += 4)
        {
            double a[4], b[4];
#pragma unroll
            for(int i = 0; i < 4; ++i)
                a[i] = sA[(k0 + q) * GEMM_LD + r0 + i * 8 + g];
#pragma unroll
            for(int i = 0; i < 4; ++i)
                b[i] = BY_COL ? sB[(c0 + i * 8 + g) * GEMM_LD + k0 + q]
                              : sB[(k0 + q) * GEMM_LD + c0 + i * 8 + g];
#pragma unroll
            for(int i = 0; i < 4; ++i)
#pragma unroll
                for(int j = 0; j < 4; ++j)
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
                                 "{%0, %1}, {%2}, {%3}, {%0, %1};\n"
                                 : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
                                 : "d"(a[i]), "d"(b[j]));
        }
    }
    template <typename F>
    __device__ __forceinline__ void each(F f)
    {
        const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
        for(int j = 0; j < 4; ++j)
#pragma unroll
            for(int e = 0; e < 2; ++e)
#pragma unroll
                for(int i = 0; i < 4; ++i)
                    f(i * 8 + g, j * 8 + q * 2 + e, acc[i][j][e]);
    }
};

template <>
struct GemmTile<float, false>
{
    float2 acc[4][4]; // rows rg*4 + i, columns cg*8 + 2p + {0, 1}
    static constexpr bool B_BY_COL = false;
    template <bool BY_COL = false>
    __device__ __forceinline__ void mma(const float* sA, const float* sB, int r0, int c0, int kk)
    {
        const int lane = threadIdx.x & 31, rg = lane & 7, cg = lane >> 3;
#pragma unroll 4
        for(int k = 0; k < kk; ++k)
        {
            const float4 a = *reinterpret_cast<const float4*>(sA + k * GEMM_LD + r0 + rg * 4);
            const float4 u0 = *reinterpret_cast<const float4*>(sB + k * GEMM_LD + c0 + cg * 8);
            const float4 u1 = *reinterpret_cast<const float4*>(sB + k * GEMM_LD + c0 + cg * 8 + 4);
            const float l[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for(int i = 0; i < 4; ++i)
            {
                fma2(acc[i][0], l[i], u0.x, u0.y);
                fma2(acc[i][1], l[i], u0.z, u0.w);
                fma2(acc[i][2], l[i], u1.x, u1.y);
                fma2(acc[i][3], l[i], u1.z, u1.w);
            }
        }
    }
    template <typename F>
    __device__ __forceinline__ void each(F f)
    {
        const int lane = threadIdx.x & 31, rg = lane & 7, cg = lane >> 3;
#pragma unroll
        for(int p = 0; p < 4; ++p)
#pragma unroll
            for(int i = 0; i < 4; ++i)
                f(rg * 4 + i, cg * 8 + 2 * p, acc[i][p].x);
#pragma unroll
        for(int p = 0; p < 4; ++p)
#pragma unroll
            for(int i = 0; i < 4; ++i)
                f(rg * 4 + i, cg * 8 + 2 * p + 1, acc[i][p].y);
    }
};

// split TF32 (the mixed solver's FP32 factorisation)
template <>
struct GemmTile<float, true>
{
    WarpTileTF32 t;
    static constexpr bool B_BY_COL = false;
    __device__ __forceinline__ void mma(const float* sA, const float* sB, int r0, int c0, int kk)
    {
        int arow[4];
#pragma unroll
        for(int i = 0; i < 4; ++i)
            arow[i] = r0 + WarpTileTF32::frag_row(i);
        for(int k0 = 0; k0 < kk; k0 += 8)
            t.mma<8>(sA + k0 * GEMM_LD, GEMM_LD, arow, sB + k0 * GEMM_LD, GEMM_LD, c0);
    }
    template <typename F>
    __device__ __forceinline__ void each(F f)
    {
        t.each(f);
    }
};

template <typename T>
struct GemmSmem
{
    T A[BLK_NB][GEMM_LD];
    T B[BLK_NB][GEMM_LD];
};

template <typename T, bool TC, bool FULL>
__device__ __forceinline__ void gemm_tile(GemmSmem<T>& sm, const LuMember<T>& M, int j0, int r0,
                                          int c0, int nr, int nc)
{
    using Tile = GemmTile<T, TC>;
    const int tid = threadIdx.x, warp = tid >> 5;
    // operands; rows and columns outside the member are zero
    if constexpr(FULL)
    {
        constexpr int V = 16 / sizeof(T), PER = 64 / V; // vectors of a column
#pragma unroll
        for(int e = tid; e < 64 * PER; e += 128)
        {
            const int i = (e % PER) * V, k = e / PER;
            cp_async16(&sm.A[k][i], &RSB_AT(M.a, r0 + i, j0 + k, M.lda, M.m, M.n));
        }
        if constexpr(Tile::B_BY_COL)
        {
#pragma unroll
            for(int e = tid; e < 64 * PER; e += 128)
            {
                const int i = (e % PER) * V, c = e / PER;
                cp_async16(&sm.B[c][i], &RSB_AT(M.a, j0 + i, c0 + c, M.lda, M.m, M.n));
            }
        }
    }
    else
    {
        for(int e = tid; e < 64 * 64; e += 128)
        {
            const int i = e & 63, k = e >> 6;
            if(i < nr)
                cp_async(&sm.A[k][i], &RSB_AT(M.a, r0 + i, j0 + k, M.lda, M.m, M.n));
            else
                sm.A[k][i] = T(0);
        }
    }
    if constexpr(!FULL || !Tile::B_BY_COL)
        for(int e = tid; e < 64 * 64; e += 128)
        {
            // FP64: 64 consecutive k of a column; else 8 k x 4 columns per warp access (whole
            // 32-byte sectors, and no bank conflict in the transposed store)
            const int k = Tile::B_BY_COL ? (e & 63) : ((e & 7) | ((e >> 4) & 0x38));
            const int c = Tile::B_BY_COL ? (e >> 6) : (((e >> 3) & 15) | ((e >> 6) & 0x30));
            T* d = Tile::B_BY_COL ? &sm.B[c][k] : &sm.B[k][c];
            if(FULL || c < nc)
                cp_async(d, &RSB_AT(M.a, j0 + k, c0 + c, M.lda, M.m, M.n));
            else
                *d = T(0);
        }
    const int wr = (warp & 1) * 32, wc = (warp >> 1) * 32;
    Tile w;
    const bool live = FULL || (wr < nr && wc < nc);
    if(live)
        w.each([&](int r, int c, auto& v) {
            v = (FULL || (wr + r < nr && wc + c < nc))
                    ? -RSB_AT(M.a, r0 + wr + r, c0 + wc + c, M.lda, M.m, M.n)
                    : T(0);
        });
    cp_async_wait();
    __syncthreads();
    if(live)
    {
        w.mma(&sm.A[0][0], &sm.B[0][0], wr, wc, BLK_NB);
        w.each([&](int r, int c, auto& v) {
            if(FULL || (wr + r < nr && wc + c < nc))
                RSB_AT(M.a, r0 + wr + r, c0 + wc + c, M.lda, M.m, M.n) = -v;
        });
    }
}

// A22 -= L21 U12 for the panel at j0: one CTA of four warps per 64 x 64 tile, K = 64 in one
// stage (a panel with fewer columns has no rows below or no columns right of it).  The tile of A22 is loaded (negated) into the accumulators while cp.async brings
// the operands in; several CTAs per SM overlap one tile's loads with another's products.
// FP64 n = 1024 x 40: 15 launches 1.36 ms, 21 TFLOP/s; FP32 split TF32 n = 256 x 2048: 3 launches
// 0.45 ms, bound by A22's traffic (1.2 GB).
template <typename T, bool TC>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 3 : 4)
    lu_gemm_kernel(LuBatch<T> L, int j0, int tiles, int tiles_m)
{
    constexpr int NB = BLK_NB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GemmSmem<T>& sm = *reinterpret_cast<GemmSmem<T>*>(smem_raw);
    LuMember<T> M;
    if(!lu_member(L, blockIdx.x / tiles, M) || lu_gave_up(L, M))
        return;
    const int t = blockIdx.x % tiles;
    const int r0 = j0 + NB + (t % tiles_m) * 64, c0 = j0 + NB + (t / tiles_m) * 64;
    const int nr = min(64, M.m - r0), nc = min(64, M.n - c0);
    // whole tiles of 16-byte aligned columns (one branch per CTA): no bounds, 16-byte copies
    const bool full = nr == 64 && nc == 64
                      && ((reinterpret_cast<uintptr_t>(M.a) | ((uintptr_t)M.lda * sizeof(T))
                           | ((uintptr_t)r0 * sizeof(T)))
                          & 15) == 0;
    if(full)
        gemm_tile<T, TC, true>(sm, M, j0, r0, c0, nr, nc);
    else
        gemm_tile<T, TC, false>(sm, M, j0, r0, c0, nr, nc);
}

// ---------------------------------------------------------------------------- L's rows
// The interchanges of all panels right of column block jblk on that block's rows: position q
// receives row perm[q], the composition of the later panels' interchanges (built from the
// last panel backwards: perm[q] = s[perm[q]] with s one panel's own map, the identity but for
// at most 128 rows).  Each column is read once and written once (FP32 n = 256 x 2048 0.21 ms).
constexpr int LEFT_NT = 256, LEFT_COLS = 32, LEFT_BUF = 32 * 1024;

template <typename T>
__global__ void __launch_bounds__(LEFT_NT)
    lu_left_kernel(LuBatch<T> L, int blocks, int max_rows)
{
    constexpr int NB = BLK_NB, PARTS = NB / LEFT_COLS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* buf = reinterpret_cast<T*>(smem_raw);
    int* perm = reinterpret_cast<int*>(smem_raw + LEFT_BUF);
    int* s = perm + max_rows;
    __shared__ int piv[NB];
    LuMember<T> M;
    if(!lu_member(L, blockIdx.x / (blocks * PARTS), M) || lu_gave_up(L, M))
        return;
    const int t = blockIdx.x % (blocks * PARTS);
    const int c0 = (t / PARTS) * NB + (t % PARTS) * LEFT_COLS;
    const int r0 = (t / PARTS + 1) * NB; // first row the later panels may move
    const int mn = min(M.m, M.n), rows = M.m - r0;
    const int tid = threadIdx.x;
    for(int q = tid; q < rows; q += LEFT_NT)
        perm[q] = s[q] = q;
    for(int j = ((mn - 1) / NB) * NB; j >= r0; j -= NB)
    {
        const int jb = min(NB, mn - j), base = j - r0;
        __syncthreads();
        if(tid < jb)
            piv[tid] = M.piv[j + tid] - 1 - j;
        __syncthreads();
        int x = -1, x0 = 0;
        if(tid < 2 * NB && (tid & (NB - 1)) < jb)
        {
            x0 = tid < NB ? tid : piv[tid - NB];
            x = x0;
#pragma unroll 8
            for(int k = jb - 1; k >= 0; --k)
            {
                const int p = piv[k];
                x = x == k ? p : (x == p ? k : x);
            }
            s[base + x0] = base + x;
        }
        __syncthreads();
        for(int q = tid; q < rows; q += LEFT_NT)
            perm[q] = s[perm[q]];
        __syncthreads();
        if(x >= 0)
            s[base + x0] = base + x0;
    }
    __syncthreads();
    const int per = max(1, min(8, (int)(LEFT_BUF / sizeof(T)) / rows)); // columns per pass
    for(int c = 0; c < LEFT_COLS; c += per)
    {
        const int nc = min(per, LEFT_COLS - c);
        for(int q = tid; q < rows; q += LEFT_NT)
        {
            T t[8];
#pragma unroll
            for(int u = 0; u < 8; ++u)
                if(u < nc)
                    t[u] = RSB_AT(M.a, r0 + q, c0 + c + u, M.lda, M.m, M.n);
#pragma unroll
            for(int u = 0; u < 8; ++u)
                if(u < nc)
                    buf[u * rows + q] = t[u];
        }
        __syncthreads();
        for(int q = tid; q < rows; q += LEFT_NT)
        {
            const int p = perm[q];
            if(p != q)
            {
#pragma unroll
                for(int u = 0; u < 8; ++u)
                    if(u < nc)
                        RSB_AT(M.a, r0 + q, c0 + c + u, M.lda, M.m, M.n) = buf[u * rows + p];
            }
        }
        __syncthreads();
    }
}

} // namespace rsb
