// cluster_step.cuh -- many time steps of 2D solves, each resident in the
// shared memory of one thread-block cluster.
//
// The grid-wide stepper (stepper.cuh) moves the field through L2 and pays a
// grid barrier per pass, about 1 us, which is most of a small grid's step; and
// it holds the whole GPU for one solve.  Here a cluster of CS CTAs holds the
// whole n x n field: CTA q has rows q R .. (q+1) R - 1 (R = n / CS) in its
// shared memory for the whole launch.  A row pass works on the CTA's own rows;
// a column pass of CTA q takes columns q R .. (q+1) R - 1, reading and writing
// them in place through distributed shared memory; a cluster barrier (a few
// hundred cycles) separates passes.  Global memory is read once at the start
// and written once at the end.  Clusters are placed by the hardware as a whole,
// so any number of solves can be queued in one launch, one cluster each, and a
// solve never waits for another.
//
// A solve's arithmetic does not depend on CS: the transforms and factors are
// per line, and a norm is formed as one compensated FP64 sum per line, in a fixed
// order over the line's threads, then summed over the lines in a fixed order by
// every CTA (blockDim is fixed per length).  So the same solve ends bit for bit the
// same whatever cluster size a batch gives it.
//
// What bounds it: about 313 instructions per point and step, issued at 0.39 to
// 0.48 per scheduler cycle with the 16 warps that fit beside the field (1024
// threads at 64 registers were no faster: 256^2 45 -> 50 us); the rest is the
// column groups' barriers and remote loads.  Batched complex64 solves on B200,
// point-steps/s of the multi-size line-pass kernel and here: 128 of 128^2 2.0e10
// -> 5.4e10, 64 of 192^2 1.75e10 -> 5.3e10, 32 of 256^2 1.9e10 -> 4.6e10, 16 of
// 384^2 1.4e10 -> 2.1e10 (7 clusters of 16 at a time); complex128 32 of 128^2
// 1.35e10 -> 3.0e10.  Slower: 8 complex64 solves, one more than fit as 16 CTAs,
// of 256^2 25 us per step in real time (23) and 48 rotating (42), of 384^2 72
// (67).  A lone solve gets 16 SMs at most: complex128 256^2 39 -> 20 us per
// step, but complex64 512^2 30 -> 55, so that one runs on the grid (batch.cu).
//
// Shared memory per CTA: the rows at a padded stride, which double as the
// exchange buffer of their own transforms; an exchange buffer for the columns
// in flight; the stage twiddles and the V/2 (x) and K (y) factor tables.
#pragma once

#include "plane.cuh"
#include "stepper.cuh"

namespace gpue {

// One solve of a batched launch (its walk lies in global memory).
struct ClusterArgs {
    PassArgs a;
    double gauge_ang[2];
    double* scal_norm;
    double* scal_guard;
    const double* target_norm;
    const double* target_guard;
    const StepPass* seq;
    int nseq;
    int pad;
};

constexpr int kClusterThreads = 512;
constexpr int kClusterMax = 16;

struct alignas(16) ClusterShared {
    double scale, guard;
    double target_norm, target_guard;
    double scratch[2 * (kClusterThreads / 32)];
};

template <typename T, int N, int RA, int RB, int RC, int P>
struct ClusterShape {
    using L = LineFFT<T, N, RA, RB, P, RC>;
    static constexpr int E = L::E;
    // (256^2 complex128: 16 lines of 16 threads, so that clusters of 8 hold it
    // with one exchange per transform: 8 solves 31.9 us per step; 8 4 8 with 512
    // threads needs clusters of 16, 40.8)
    static constexpr int MOST = sizeof(T) == 8 && N == 256 ? 256 : kClusterThreads;
    static constexpr int THREADS = N * P < MOST ? N * P : MOST;
    static constexpr int LPR = THREADS / P;  // lines in flight
    static constexpr int PHYS = L::phys(N - 1) + 1;
    // row stride: lines of 8 threads share a half-warp, so offset them by half
    // a bank row
    static constexpr int XS = (PHYS + 15) / 16 * 16 + (P == 8 ? 8 : 0);
    // column stride: lanes are (column, thread) with up to 8 adjacent columns,
    // spread over the banks by an odd or small even offset
    static constexpr int LSC = (PHYS + 15) / 16 * 16 + (sizeof(T) == 4 ? 2 : 1);
    static constexpr size_t TW = (size_t)L::kStageTableLen * 16;
    static constexpr size_t FACB = (size_t)N * 2 * sizeof(T);
    static size_t smem(int cs) {
        const int R = (N + cs - 1) / cs;
        return sizeof(ClusterShared) + sizeof(ClusterArgs) + TW + 2 * FACB + (size_t)N * 16 +
               (size_t)THREADS * 8 + (size_t)R * XS * sizeof(cx<T>) +
               (size_t)LPR * LSC * sizeof(cx<T>) + 64;
    }
};

template <typename T>
__device__ __forceinline__ void dsmem_store(unsigned addr, cx<T> v) {
    if constexpr (sizeof(T) == 4)
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y)
                     : "memory");
    else
        asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y)
                     : "memory");
}
__device__ __forceinline__ double2 dsmem_load_f64x2(unsigned addr) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];"
                 : "=d"(v.x), "=d"(v.y)
                 : "r"(addr)
                 : "memory");
    return v;
}
__device__ __forceinline__ unsigned cluster_ctas() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

template <typename T, int N, int RA, int RB, int RC, int P, bool REAL, class Args>
__device__ __forceinline__ void cluster_steps(const Args& s, const StepPass* __restrict__ seq,
                                              ClusterShared* sh, unsigned char* p) {
    using S_ = ClusterShape<T, N, RA, RB, RC, P>;
    using L = typename S_::L;
    using Fac = std::conditional_t<std::is_same<T, float>::value, float2, double2>;
    constexpr int E = S_::E;
    constexpr int gstate = REAL ? 1 : 0;
    const PassArgs& a = s.a;
    const int tid = threadIdx.x;
    const int CS = (int)cluster_ctas(), rank = (int)cluster_rank();
    const int R = (N + CS - 1) / CS;                 // rows (then columns) per CTA
    const int first = rank * R;
    const int mine = min(R, N - first);              // of which this CTA has
    const unsigned Rmul = (unsigned)((0x100000000ull + R - 1) / R);  // y / R by high product

    cx<T>* tw_s = reinterpret_cast<cx<T>*>(p);
    p += S_::TW;
    Fac* vx_s = reinterpret_cast<Fac*>(p);
    p += S_::FACB;
    Fac* ky_s = reinterpret_cast<Fac*>(p);
    p += S_::FACB;
    double2* line_s = reinterpret_cast<double2*>(p);  // [N]: (sum, compensation) of this CTA's lines
    p += (size_t)N * 16;
    double* part_s = reinterpret_cast<double*>(p);  // [THREADS]
    p += (size_t)S_::THREADS * 8;
    cx<T>* X = reinterpret_cast<cx<T>*>(p);  // [R][XS]
    p += (size_t)R * S_::XS * sizeof(cx<T>);
    cx<T>* S = reinterpret_cast<cx<T>*>(p);  // [LPR][LSC]

    if constexpr (std::is_same<T, float>::value) {
        L::build_stage_table(reinterpret_cast<float4*>(tw_s), static_cast<const float4*>(a.tw),
                             tid, S_::THREADS);
        for (int i = tid; i < N; i += S_::THREADS) vx_s[i] = a.vd[0][i], ky_s[i] = a.kd[1][i];
    } else {
        L::build_stage_table(reinterpret_cast<double2*>(tw_s),
                             static_cast<const double2*>(a.tw), tid, S_::THREADS);
        for (int i = tid; i < N; i += S_::THREADS) vx_s[i] = a.vfac[0][i], ky_s[i] = a.kfac[1][i];
    }
    if (tid == 0) {
        sh->scale = *s.scal_norm;
        sh->guard = *s.scal_guard;
        sh->target_norm = *s.target_norm;
        sh->target_guard = *s.target_guard;
    }
    const cx<T>* in = static_cast<const cx<T>*>(a.in);
    for (int i = tid; i < mine * N; i += S_::THREADS) {
        const int r = i / N, x = i % N;
        X[r * S_::XS + L::phys(x)] = in[(size_t)(first + r) * N + x];
    }
    __syncthreads();
    cluster_arrive();
    cluster_wait();

    // rows: a line's P threads are adjacent.  columns: groups of cg adjacent
    // columns (cg P threads, whole warps, at one named barrier), lanes along x
    int cgs = 3;
    if (P == 64) cgs = 2;
    while (cgs > 0 && ((1 << cgs) > mine) && ((P << (cgs - 1)) % 32 == 0)) --cgs;
    const int gthreads = P << cgs, grp = tid / gthreads;
    const int tr = tid & (P - 1), lr = tid / P;
    const int tc = ((tid % gthreads) >> cgs) & (P - 1);
    const int lc = (grp << cgs) + (tid & ((1 << cgs) - 1));
    const unsigned xbase = smem_addr(X);

    StepPass sp = seq[0];
    for (int k = 0; k < s.nseq; ++k) {
        const bool colpass = sp.flags & SP_COL;
        const int t = colpass ? tc : tr, l0 = colpass ? lc : lr;
        const bool norm = sp.flags & (SP_NORM | SP_GUARD);
        for (int base = 0; base < R; base += S_::LPR) {
            // whole warps (rows) or whole barrier groups (columns) past the
            // CTA's lines leave the round
            const int l = base + l0;
            const int lw = colpass ? base + (grp << cgs) : base + (tid & ~31) / P;
            if (lw >= mine) {
                if (norm) __syncthreads();
                if (norm) __syncthreads();
                continue;
            }
            const bool ok = l < mine;
            const int g = first + (ok ? l : 0);  // the line in the field
            // (a thread past the CTA's lines works on scratch and stores nothing)
            cx<T>* sl = colpass || !ok ? S + l0 * S_::LSC : X + l * S_::XS;
            auto sync = [&] {
                if (colpass) {
                    asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(gthreads) : "memory");
                } else if constexpr (P <= 32) {
                    __syncwarp();
                } else {
                    asm volatile("bar.sync %0, %1;" ::"r"(1 + lr), "n"(P) : "memory");
                }
            };
            auto remote = [&](int e) {
                const unsigned y = (unsigned)L::index(t, e);
                const unsigned q = __umulhi(y, Rmul);
                return dsmem_map(xbase + ((y - q * R) * S_::XS + L::phys(g)) * sizeof(cx<T>), q);
            };
            cx<T> v[E];
            if (colpass) {
#pragma unroll
                for (int e = 0; e < E; ++e) v[e] = dsmem_load<T>(remote(e));
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) v[e] = sl[L::phys(L::index(t, e))];
                sync();  // the row is read before its exchanges write it
            }
            KSum acc{0.0, 0.0};
            for (unsigned ops = sp.ops; ops; ops >>= 4) {
                const bool conj = !std::is_same<T, float>::value && (ops & 15u) == OP_FFT_I;
                if (conj) {
#pragma unroll
                    for (int e = 0; e < E; ++e) v[e].y = -v[e].y;
                }
                switch (conj ? (unsigned)OP_FFT_F : ops & 15u) {
                    case OP_FFT_F:
                        L::template forward<true, false>(v, t, sl, tw_s, sync);
                        break;
                    case OP_FFT_I:
                        if constexpr (std::is_same<T, float>::value)
                            L::template forward<true, true>(v, t, sl, tw_s, sync);
                        break;
                    case OP_SCALE: {
                        const T f = (T)sh->scale;
#pragma unroll
                        for (int e = 0; e < E; ++e) v[e] = cscale(v[e], f);
                        break;
                    }
                    case OP_VHALF: {
                        const cx<double> lf = ld2(a.vfac[1], g);
                        if constexpr (std::is_same<T, float>::value)
                            op_vhalf_f32<L>(v, t, vx_s, line_delta(lf), a, gstate, a.nl_coef);
                        else
                            op_vhalf_sep<T, L>(v, t, vx_s, lf, a, gstate, a.nl_coef);
                        break;
                    }
                    case OP_KPHASE: {
                        const cx<double> lf = ld2(a.kfac[0], g);
                        const double ks =
                            (sp.flags & SP_KGUARD) ? a.kscale * sh->guard : a.kscale;
                        if constexpr (std::is_same<T, float>::value)
                            op_kphase_f32<L>(v, t, ky_s, line_delta(lf), (float)ks);
                        else
                            op_kphase_f64<L>(v, t, ky_s, cscale(lf, ks), gstate);
                        break;
                    }
                    case OP_GAUGE: {
                        const double ang =
                            (colpass ? s.gauge_ang[1] : s.gauge_ang[0]) * a.pos[colpass ? 0 : 1][g];
                        op_gauge<T, L>(v, gauge_consts<L>(t, ang, gstate, a.gscale), gstate);
                        break;
                    }
                    case OP_NORM:
                        if constexpr (std::is_same<T, float>::value) op_norm_f32<E>(v, acc);
                        else op_norm<T, E>(v, acc);
                        break;
                    default:
                        break;
                }
                if (conj) {
#pragma unroll
                    for (int e = 0; e < E; ++e) v[e].y = -v[e].y;
                }
            }
            if (ok) {
                if (colpass) {
#pragma unroll
                    for (int e = 0; e < E; ++e) dsmem_store<T>(remote(e), v[e]);
                } else {
#pragma unroll
                    for (int e = 0; e < E; ++e) sl[L::phys(L::index(t, e))] = v[e];
                }
            }
            if (norm) {
                // one compensated sum per line, in the order of its threads
                __syncthreads();  // the previous round's sums are read
                part_s[l0 * P + t] = acc.s + acc.c;  // (one term: exact)
                __syncthreads();
                KSum q{part_s[tid], 0.0};
                if constexpr (P > 32) {
                    if (tr < 32) q.add(part_s[tid + 32]);
                }
#pragma unroll
                for (int o = (P < 32 ? P : 32) / 2; o > 0; o >>= 1) {
                    const double os = __shfl_down_sync(0xffffffffu, q.s, o, P < 32 ? P : 32);
                    const double oc = __shfl_down_sync(0xffffffffu, q.c, o, P < 32 ? P : 32);
                    q.merge(os, oc);
                }
                if (tr == 0 && base + lr < mine) line_s[base + lr] = make_double2(q.s, q.c);
            }
        }
        const unsigned flags = sp.flags;
        if (k + 1 < s.nseq) sp = seq[k + 1];
        __syncthreads();
        cluster_arrive();
        cluster_wait();
        if (norm) {
            // every CTA sums all lines in the same order; line_s is written
            // again only after the next cluster barrier
            KSum r{0.0, 0.0};
            for (int i = tid; i < N; i += S_::THREADS) {
                const unsigned q = __umulhi((unsigned)i, Rmul);
                const double2 ls = dsmem_load_f64x2(dsmem_map(smem_addr(line_s) + (i - q * R) * 16, q));
                r.merge(ls.x, ls.y);
            }
            r = block_reduce(r, sh->scratch);
            if (tid == 0) {
                const double sum = r.s + r.c;
                if (flags & SP_NORM) sh->scale = sqrt(sh->target_norm / sum);
                else sh->guard = sqrt(sh->target_guard / sum);
            }
            __syncthreads();
        }
    }
    cx<T>* out = static_cast<cx<T>*>(a.out);
    for (int i = tid; i < mine * N; i += S_::THREADS) {
        const int r = i / N, x = i % N;
        out[(size_t)(first + r) * N + x] = X[r * S_::XS + L::phys(x)];
    }
    if (rank == 0 && tid == 0) {
        *s.scal_norm = sh->scale;
        *s.scal_guard = sh->guard;
    }
    // no CTA leaves while another may still read its line sums
    cluster_arrive();
    cluster_wait();
}

// One solve, the walk in the kernel's parameters.
template <typename T, int N, int RA, int RB, int RC, int P, bool REAL>
__global__ void __launch_bounds__(ClusterShape<T, N, RA, RB, RC, P>::THREADS, 1)
    k_cluster_one(const __grid_constant__ StepArgs s) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterShared* sh = reinterpret_cast<ClusterShared*>(smem_raw);
    cluster_steps<T, N, RA, RB, RC, P, REAL>(s, s.seq, sh, smem_raw + sizeof(ClusterShared));
}

// Many solves: cluster q runs many[q].
template <typename T, int N, int RA, int RB, int RC, int P, bool REAL>
__global__ void __launch_bounds__(ClusterShape<T, N, RA, RB, RC, P>::THREADS, 1)
    k_cluster_many(const ClusterArgs* __restrict__ many) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterShared* sh = reinterpret_cast<ClusterShared*>(smem_raw);
    ClusterArgs* s = reinterpret_cast<ClusterArgs*>(smem_raw + sizeof(ClusterShared));
    const ClusterArgs* g = many + cluster_index();
    if (g->a.active && *g->a.active == 0) return;  // converged: the whole cluster leaves
    static_assert(sizeof(ClusterArgs) % 4 == 0, "copied by words");
    for (int i = threadIdx.x; i < (int)(sizeof(ClusterArgs) / 4); i += blockDim.x)
        reinterpret_cast<unsigned*>(s)[i] = reinterpret_cast<const unsigned*>(g)[i];
    __syncthreads();
    cluster_steps<T, N, RA, RB, RC, P, REAL>(
        *s, s->seq, sh, smem_raw + sizeof(ClusterShared) + (sizeof(ClusterArgs) + 15) / 16 * 16);
}

// A compiled cluster stepper: shared memory by cluster size, the kernels by
// time kind (void* keeps the launch attributes with the caller).
struct ClusterKernel {
    int n, ra, rb, rc, p;
    int threads;
    size_t (*smem)(int cs);
    const void* one[2];
    const void* many[2];
};
const ClusterKernel* find_cluster_kernel(int prec, int n);
const ClusterKernel* cluster_table_f32(int* count);
const ClusterKernel* cluster_table_f64(int* count);

#define GPUE_CLUSTER(T, N, RA, RB, RC, P)                                                   \
    ClusterKernel{N, RA, RB, RC, P, ClusterShape<T, N, RA, RB, RC, P>::THREADS,              \
                  &ClusterShape<T, N, RA, RB, RC, P>::smem,                                  \
                  {(const void*)&k_cluster_one<T, N, RA, RB, RC, P, false>,                  \
                   (const void*)&k_cluster_one<T, N, RA, RB, RC, P, true>},                  \
                  {(const void*)&k_cluster_many<T, N, RA, RB, RC, P, false>,                 \
                   (const void*)&k_cluster_many<T, N, RA, RB, RC, P, true>}}

}  // namespace gpue
