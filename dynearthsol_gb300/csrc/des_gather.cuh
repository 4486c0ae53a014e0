// des_gather.cuh -- node sums over the support lists, in ascending element
// order (the reference's serial order, whatever the kernel's shape).
//
// Two shapes of the same sums, with the same terms in the same order and so
// the same bits:
// * walk: a thread per node goes through its ~24 support entries.  A large
//   mesh fills the GPU with nodes, whose warps hide one another's loads.
// * staged: a block takes NPB consecutive nodes, whose entries are one
//   contiguous range of the support lists.  All its threads form the terms
//   of that range, an entry each, and stage them in shared memory; then a
//   thread per (quantity, node) adds its node's terms.  On a small mesh the
//   walk is a chain of 24 dependent pairs of loads on a few SMs; here the
//   entries' loads and arithmetic run side by side on eight times as many
//   threads.  The range is staged in chunks of CAP entries, so a node of any
//   degree (and any mix of degrees) is summed.
// node_staged() draws the line.
#pragma once
#include <type_traits>

#include <cuda_runtime.h>

#include "des_common.cuh"
#include "des_dw.cuh"

namespace des {

constexpr int NPB = 8, STAGED_THREADS = 192;

// p: the launch's context, n: its nodes.  Staging pays while the walk would
// put too few warps on each SM to hide its chain of loads; beyond about a wave
// of blocks it only adds the trip through shared memory.  The lines lie where
// the two take the same time, at 56 nodes per SM with FP64 sums and at 160 with
// the double-word sums of a mixed context, whose additions cost the few adding
// threads less.  Measured, staged / walk:
// * FP64, 200 steps in 2D: 12,000 triangles (6,191 nodes) 7.7 / 8.1 ms, 16,000
//   (8,241) 8.1 / 8.1, 24,000 (12,291) 10.5 / 8.9, 36,000 (18,361) 12.1 / 9.8;
//   100 steps in 3D: 14,400 tets (3,087 nodes) 6.2 / 7.3, 42,336 (8,410) 11.0 /
//   11.6, 56,448 (10,933) 13.1 / 13.1, 73,728 (14,157) 16.7 / 15.9; windows of
//   20 steps and their reverse: 14,400 tets 3.95 / 4.55, 42,336 6.14 / 6.16,
//   73,728 8.47 / 8.01.
// * mixed, 100 steps: 73,728 tets 6.90 / 7.74 ms, 121,296 (22,815 nodes) 10.03 /
//   10.14, 134,400 (25,215) 10.78 / 10.57, 162,624 (30,375) 13.36 / 12.64.
// 192 threads take the entries of 8 nodes (~24 each) in one chunk: 100 steps of
// a 648-tet mesh, with the state's copies, 5.83 ms, 5.98 ms with 96 threads.
inline bool node_staged_fp64(long long n) { return n <= 152LL * 56; }
inline bool node_staged(const KP &p, long long n) { return p.shpdw ? n <= 152LL * 160 : node_staged_fp64(n); }

// The sums' arithmetic: a quantity's term, state, addition and value.
struct SumF64 {   // FP64 additions
    using Term = double;
    using State = double;
    static __device__ __forceinline__ void add(int, State &s, Term t) { s += t; }
    static __device__ __forceinline__ double value(int, const State &s) { return s; }
};
struct SumDw {    // compensated FP32 sums of double-word terms (des_dw.cuh)
    using Term = float2;
    using State = dw_sum;
    static __device__ __forceinline__ void add(int, State &s, Term t) { s.add(dw_of2(t)); }
    static __device__ __forceinline__ double value(int, const State &s) { return s.value(); }
};
struct SumDwAcc { // double-word additions of double-word terms, accurate under cancellation
    using Term = float2;
    using State = dw;
    static __device__ __forceinline__ void add(int, State &s, Term t) { s = dw_add(s, dw_of2(t)); }
    static __device__ __forceinline__ double value(int, const State &s) { return f64_of(s); }
};

__device__ __forceinline__ float2 pair_of(dw w) { return make_float2(w.hi, w.lo); }

// One quantity's staged terms.  A slot in 128 bytes is left out, so that the
// threads of a warp, 24 entries apart, read different banks.
template <class T, int CAP>
struct Staged {
    static constexpr int ROW = 128 / (int)sizeof(T);
    T v[CAP + CAP / ROW + 1];
    __device__ __forceinline__ T &operator[](int r) { return v[r + r / ROW]; }
};

template <class P, class Term>
__device__ __forceinline__ void entry_terms(Term &term, int q, typename P::Term *t, int n)
{
    if constexpr (std::is_invocable_v<Term, int, typename P::Term *, int>) term(q, t, n);
    else term(q, t);
}

// The sums of NQ quantities over the support of the nodes [lo, hi) of a
// launch, by the calling kernel's whole grid: term(q, t) or term(q, t, n) forms
// the NQ terms of support entry q (n: its node in a walk; entries staged side by
// side are not told); first(c, n) is the value that quantity c of node n
// starts from.  Returns the node whose NQ sums the thread holds in out, or -1
// when it holds none.  Every thread of the block calls it; of the NQ sums, the
// first nq are formed and the others hold nothing.
template <class P, int NQ, int ND, bool STAGED, class Term, class First>
__device__ __forceinline__ int node_sums(const int *__restrict__ off, int lo, int hi, int nq, Term term, First first,
                                         double *out)
{
    if constexpr (!STAGED) {
        const int n = lo + blockIdx.x * blockDim.x + threadIdx.x;
        if (n >= hi) return -1;
        typename P::State s[NQ];
#pragma unroll
        for (int c = 0; c < NQ; ++c) s[c] = first(c, n);
        for (int q = off[n]; q < off[n + 1]; ++q) {
            typename P::Term t[NQ];
            entry_terms<P>(term, q, t, n);
#pragma unroll
            for (int c = 0; c < NQ; ++c)
                if (c < nq) P::add(c, s[c], t[c]);
        }
#pragma unroll
        for (int c = 0; c < NQ; ++c) out[c] = P::value(c, s[c]);
        return n;
    } else {
        constexpr int CAP = NPB * (ND == 3 ? 28 : 8);   // interior degrees 24 and 6, with some room
        __shared__ Staged<typename P::Term, CAP> slot[NQ];
        __shared__ double sum[NQ][NPB];
        const int n0 = lo + blockIdx.x * NPB, nb = min(NPB, hi - n0);
        if (nb <= 0) return -1;
        const int i = threadIdx.x % NPB, c = threadIdx.x / NPB;
        const int q0 = off[n0], q1 = off[n0 + nb];
        int a = q1, b = q1;
        typename P::State s{};
        if (c < nq && i < nb) {
            a = off[n0 + i];
            b = off[n0 + i + 1];
            s = first(c, n0 + i);
        }
        for (int base = q0; base < q1; base += CAP) {
            const int end = min(base + CAP, q1);
            for (int q = base + (int)threadIdx.x; q < end; q += STAGED_THREADS) {
                typename P::Term t[NQ];
                entry_terms<P>(term, q, t, -1);
#pragma unroll
                for (int k = 0; k < NQ; ++k)
                    if (k < nq) slot[k][q - base] = t[k];
            }
            __syncthreads();
            const int last = min(b, end);
            for (int q = max(a, base); q < last; ++q) P::add(c, s, slot[c][q - base]);
            if (end < q1) __syncthreads();   // the next chunk overwrites the slots
        }
        if (c < NQ && i < nb) sum[c][i] = P::value(c, s);
        __syncthreads();
        if (threadIdx.x >= nb) return -1;
#pragma unroll
        for (int k = 0; k < NQ; ++k) out[k] = sum[k][threadIdx.x];
        return n0 + threadIdx.x;
    }
}

// sums that start from zero
template <class P>
struct FromZero {
    __device__ __forceinline__ typename P::State operator()(int, int) const { return typename P::State{}; }
};

// KERNEL<..., STAGED> over n nodes of the context p on stream s; KERNEL names
// the template argument STAGED where it takes the shape
#define DES_NODES(KERNEL, n, s, ...) DES_NODES_IF(des::node_staged(p, (n)), KERNEL, n, s, __VA_ARGS__)
#define DES_NODES_IF(IN_BLOCKS, KERNEL, n, s, ...)                                                                    \
    do {                                                                                                              \
        const long long n_ = (n);                                                                                     \
        if (IN_BLOCKS) {                                                                                              \
            constexpr bool STAGED = true;                                                                             \
            KERNEL<<<(int)std::max(1LL, (n_ + des::NPB - 1) / des::NPB), des::STAGED_THREADS, 0, (s)>>>(__VA_ARGS__); \
        } else {                                                                                                      \
            constexpr bool STAGED = false;                                                                            \
            DES_LAUNCH(KERNEL, n_, (s), __VA_ARGS__);                                                                 \
        }                                                                                                             \
    } while (0)

}  // namespace des
