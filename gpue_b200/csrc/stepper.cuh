// stepper.cuh -- many time steps of 2D solves in one cooperative launch.
//
// A 2D step is a chain of row and column passes (the schedules of engine.cu)
// that each need the whole field of the one before.  Launched one by one they
// cost 4 to 5 us each whatever the grid: launch and drain, cold instruction
// caches, operator constants formed anew.  Here every CTA owns one tile of C
// rows and one tile of C columns of its solve for the whole launch and walks
// the passes of up to kStepMaxSeq entries, with a grid barrier where a pass
// reads what other CTAs wrote:
//
//   - the field moves between passes through global memory (it stays in L2;
//     loads and stores bypass L1);
//   - consecutive row passes (the renormalisation lies between them in
//     imaginary time) keep the rows in registers; only the norm crosses CTAs;
//   - twiddles (the per-stage table) and the per-axis factors sit in shared
//     memory, the line factors and the gauge constants of the CTA's own lines
//     are formed once per launch;
//   - reductions: every CTA leaves its compensated FP64 partial with the pass's
//     number in one 16-byte slot, and every CTA reads all slots and sums them in
//     the same order, so all hold the same factor after one hop and no barrier.
//
// Barriers wait on CTAs of the same launch only, which a cooperative launch
// makes resident together.  Every wait is bounded in time: one that gives up
// sets *err, the CTA leaves the walk, and so do the others when their own wait
// runs out.
//
// What bounds it, and the shapes.  A pass is latency: at 256^2 complex128 it
// takes about 780 cycles to load, 2200 to transform twice, 1900 in the barrier
// and 1800 per norm; at 1024^2 complex64 the SMs with most lines issue 85 % of
// their cycles.  So the lines are dealt out as one CTA per SM (C a divisor of n,
// at least n/148) where a line has at most 32 threads; lines of 64 threads run as
// several smaller CTAs per SM, whose column barriers then stop 2 to 8 warps
// instead of all (1024^2 complex64: 42 us per step as 256 CTAs of 4 lines, 48
// with 7 lines and 147 CTAs).  Time per step on B200, as line passes before this
// kernel and now: complex128 128^2 15.3 -> 8.5 us, 256^2 15.7 -> 9.0, 320^2 (real
// time) 27.4 -> 12.2, 384^2 rotating 34.2 -> 21.4, 768^2 42.8 -> 27.9, 1024^2
// rotating 68.2 -> 59.4; complex64 256^2 13.3 -> 8.1, 640^2 35.8 -> 19.7, 768^2
// 31.3 -> 22.2, 1024^2 rotating 47.6 -> 39.7.
#pragma once

#include <type_traits>

#include "pass.cuh"

namespace gpue {

constexpr int kStepMaxSeq = 1280;
constexpr unsigned long long kStepWaitNs = 4000000000ull;  // a wait gives up after 4 s

// One pass of the walk: up to 8 op codes (4 bits each, first in the low bits)
// and its flags.
struct StepPass {
    unsigned ops;
    unsigned flags;
};
enum : unsigned {
    SP_COL = 1,       // columns (axis 1), else rows (axis 0)
    SP_LOAD = 2,      // read the lines (else they are still in registers)
    SP_STORE = 4,     // write them back
    SP_NORM = 8,      // ends with a norm: its factor is the next OP_SCALE's
    SP_GUARD = 16,    // ends with a norm: its factor scales later K passes
    SP_KGUARD = 32,   // the K factor takes the guard factor
    SP_SYNC = 64,     // all CTAs finish this pass before the next
};

struct StepArgs {
    PassArgs a;            // field, tables and constants (per-pass fields unused)
    double gauge_ang[2];   // gauge angle per momentum index and unit position, x and y pass
    unsigned* sync;        // [0] barrier count, [1] CTAs finished; zero between launches
    double2* slots;        // one per CTA (slot_store); zero between launches
    double* scal_norm;     // the renormalisation factor, read at the start, written at the end
    double* scal_guard;
    const double* target_norm;
    const double* target_guard;
    int* err;
    unsigned long long wait_ns;  // a wait gives up after this long
    unsigned more_ctas;          // barriers wait for, norms ask for: 0, or (GPUE_TEST_STEP_WAIT,
    unsigned more_passes;        // tests only) more than ever come, so every such wait runs out
    int nseq;
    StepPass seq[kStepMaxSeq];
};

// The shared-memory image of a team's constants.
struct alignas(16) StepShared {
    double scale, guard;
    double target_norm, target_guard;
    int abort;
    unsigned more_passes;
    unsigned long long wait_ns;
    double scratch[2 * (512 / 32)];
};

template <typename T, int N, int RA, int RB, int RC, int P, int C>
struct StepShape {
    using L = LineFFT<T, N, RA, RB, P, RC>;
    static constexpr int E = L::E;
    // (else a thread of the last CTA could own a row but no column, and what the
    // one left in its registers would enter the other's norm)
    static_assert(N % C == 0, "every CTA holds C whole rows and C whole columns");
    // line stride: the C columns a warp touches at once (16 or 8 lanes at a time)
    // on distinct banks
    static constexpr int W = sizeof(T) == 4 ? 16 : 8;
    static constexpr int C2 = C <= 1 ? 1 : C <= 2 ? 2 : C <= 4 ? 4 : C <= 8 ? 8 : 16;
    static constexpr int LS = L::kPad16 + (W / C2 > 1 ? W / C2 : 1);
    // the per-stage twiddle table and the V/2 (x) and K (y) factors: 1024
    // complex128 points leave no room for the factors beside the exchange
    static constexpr bool FAC = sizeof(T) == 4 || N <= 768;
    // two exchange buffers (one barrier per exchange instead of two) where they fit
    static constexpr int NBUF = sizeof(T) == 4 || N <= 640 ? 2 : 1;
    static constexpr size_t TW = (size_t)L::kStageTableLen * 16;
    static constexpr size_t FACB = FAC ? (size_t)N * 2 * sizeof(T) : 0;  // one factor table
    static constexpr size_t fixed_bytes() { return sizeof(StepShared) + TW + 2 * FACB; }
    // per thread: W^t of the two gauge passes; per line: A, B, W^(-n/2) of both
    static size_t smem(int) {
        return fixed_bytes() + (size_t)NBUF * C * LS * sizeof(cx<T>) + (size_t)C * P * 32 +
               (size_t)C * 96;
    }
};

__device__ __forceinline__ uint64_t step_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// All CTAs of the team arrive and wait; false when the wait ran out.
__device__ __forceinline__ bool step_barrier(unsigned* count, unsigned target, StepShared* sh) {
    __syncthreads();  // every thread's stores before thread 0's release
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        unsigned v, polls = 0;
        uint64_t t0 = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
            if (v >= target) break;
            if ((++polls & 1023u) == 0u) {
                const uint64_t now = step_ns();
                if (t0 == 0) t0 = now;
                else if (now - t0 > sh->wait_ns) {
                    sh->abort = 1;
                    break;
                }
            }
        }
    }
    __syncthreads();
    return sh->abort == 0;
}

// A slot is written and read as one 16-byte access, so a reader that sees the
// pass number sees the partial of that pass: the sum, and its compensation with
// the pass number in the low 16 of its 52 fraction bits (the compensation is at
// most 2^-53 of the sum, so they stand below 2^-89 of it).
constexpr unsigned long long kSlotPass = 0xffffull;
static_assert(kStepMaxSeq < (int)kSlotPass, "pass numbers fit a slot");
__device__ __forceinline__ void slot_store(double2* p, KSum v, unsigned pass) {
    const unsigned long long c =
        ((unsigned long long)__double_as_longlong(v.c) & ~kSlotPass) | pass;
    asm volatile(
        "{ .reg .b128 q; mov.b128 q, {%1, %2}; st.relaxed.gpu.global.b128 [%0], q; }" ::"l"(p),
        "l"(__double_as_longlong(v.s)), "l"(c)
        : "memory");
}
__device__ __forceinline__ unsigned slot_load(const double2* p, KSum& v) {
    long long a;
    unsigned long long c;
    asm volatile("{ .reg .b128 q; ld.relaxed.gpu.global.b128 q, [%2]; mov.b128 {%0, %1}, q; }"
                 : "=l"(a), "=l"(c)
                 : "l"(p)
                 : "memory");
    v.s = __longlong_as_double(a);
    v.c = __longlong_as_double((long long)(c & ~kSlotPass));
    return (unsigned)(c & kSlotPass);
}

// The sum of all CTAs' partials of a pass, in a fixed order, by one warp: a
// lane reads its slots in one batch until all carry the pass's number.
__device__ __forceinline__ double slots_sum(const double2* slots, int n, unsigned pass,
                                            StepShared* sh) {
    constexpr int B = 5;  // 148 CTAs in one batch
    const int lane = threadIdx.x & 31;
    KSum r{0.0, 0.0};
    uint64_t t0 = 0;
    for (int first = lane; first < n; first += 32 * B) {
        KSum q[B];
        unsigned polls = 0;
        for (;;) {
            bool ready = true;
#pragma unroll
            for (int b = 0; b < B; ++b) {
                q[b] = KSum{0.0, 0.0};
                if (first + 32 * b < n) ready &= slot_load(slots + first + 32 * b, q[b]) == pass;
            }
            if (ready) break;
            if ((++polls & 1023u) == 0u) {
                const uint64_t now = step_ns();
                if (t0 == 0) t0 = now;
                else if (now - t0 > sh->wait_ns) {
                    sh->abort = 1;
                    break;
                }
            }
        }
#pragma unroll
        for (int b = 0; b < B; ++b) r.merge(q[b].s, q[b].c);
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double os = __shfl_down_sync(0xffffffffu, r.s, o);
        const double oc = __shfl_down_sync(0xffffffffu, r.c, o);
        r.merge(os, oc);
    }
    return r.s + r.c;
}

// TAB: full-field V and gauge tables (a.vtab, a.atab) in place of the
// separable potential and the rotation preset.
template <typename T, int N, int RA, int RB, int RC, int P, bool TAB, bool REAL, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    k_step2d(const __grid_constant__ StepArgs s) {
    using S_ = StepShape<T, N, RA, RB, RC, P, MAXT / P>;
    using L = typename S_::L;
    using Fac = std::conditional_t<std::is_same<T, float>::value, float2, double2>;
    constexpr int E = S_::E;
    constexpr int gstate = REAL ? 1 : 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    StepShared* sh = reinterpret_cast<StepShared*>(smem_raw);
    const int tid = threadIdx.x, nthreads = blockDim.x;
    const int C = nthreads / P;

    const PassArgs& a = s.a;
    const int ncta = (int)gridDim.x, rank = (int)blockIdx.x;
    // a converged solve of a batched run: every CTA leaves before the first barrier
    if (a.active && *a.active == 0) return;

    // shared memory: StepShared | stage twiddles | V/2 x, K y factors |
    // exchange | W^t of both gauge passes | their line constants
    unsigned char* p = smem_raw + sizeof(StepShared);
    cx<T>* tw_s = reinterpret_cast<cx<T>*>(p);
    p += S_::TW;
    Fac* vx_s = reinterpret_cast<Fac*>(p);
    Fac* ky_s = vx_s + (S_::FAC ? N : 0);
    p += 2 * S_::FACB;
    cx<T>* xch = reinterpret_cast<cx<T>*>(p);
    p += (size_t)S_::NBUF * C * S_::LS * sizeof(cx<T>);
    cx<double>* gt_s = reinterpret_cast<cx<double>*>(p);  // [2][threads]
    cx<double>* gl_s = gt_s + 2 * nthreads;               // [2][C][3]

    if constexpr (std::is_same<T, float>::value)
        L::build_stage_table(reinterpret_cast<float4*>(tw_s), static_cast<const float4*>(a.tw),
                             tid, nthreads);
    else
        L::build_stage_table(reinterpret_cast<double2*>(tw_s),
                             static_cast<const double2*>(a.tw), tid, nthreads);
    const Fac *vx, *ky;
    if constexpr (std::is_same<T, float>::value) vx = a.vd[0], ky = a.kd[1];
    else vx = a.vfac[0], ky = a.kfac[1];
    if constexpr (S_::FAC) {
        for (int i = tid; i < N; i += nthreads) {
            vx_s[i] = vx[i];
            ky_s[i] = ky[i];
        }
        vx = vx_s;
        ky = ky_s;
    }
    if (tid == 0) {
        sh->abort = 0;
        sh->more_passes = s.more_passes;
        sh->wait_ns = s.wait_ns;
        sh->scale = *s.scal_norm;
        sh->guard = *s.scal_guard;
        sh->target_norm = *s.target_norm;
        sh->target_guard = *s.target_guard;
    }

    // thread (line, place in the line) for rows (places adjacent) and columns
    // (lines adjacent, so a warp reads whole row segments)
    const int tr = tid % P, cr = tid / P;
    const int cc = tid % C, tc = tid / C;
    const int row = rank * C + cr, col = rank * C + cc;
    // the other axis' factors at the CTA's own row and column
    const cx<double> lfv = ld2(a.vfac[1], row);
    const cx<double> lfk = ld2(a.kfac[0], col);
    // the rotation gauge's angles per momentum index along the row and column
    const double ang[2] = {s.gauge_ang[0] * a.pos[1][row], s.gauge_ang[1] * a.pos[0][col]};
    if constexpr (!TAB) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            if (s.gauge_ang[g] == 0.0) continue;
            const int t = g ? tc : tr, c = g ? cc : cr;
            const GaugeConsts gc = gauge_consts<L>(t, ang[g], gstate, a.gscale);
            gt_s[g * nthreads + tid] = gc.wt;
            if (t == 0) {
                cx<double>* gl = gl_s + (g * C + c) * 3;
                gl[0] = gc.wa;
                gl[1] = gc.wb;
                gl[2] = gc.wh;
            }
        }
    }
    __syncthreads();

    cx<T> v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = cx<T>{(T)0, (T)0};
    unsigned target = s.more_ctas;
    StepPass sp = s.seq[0];
    for (int k = 0; k < s.nseq; ++k) {
        const bool colpass = sp.flags & SP_COL;
        // (the mask changes nothing: it lets the compiler fold the exchange offsets)
        const int t = (colpass ? tc : tr) & (P - 1);
        const int c = colpass ? cc : cr;
        cx<T>* sl = xch + c * S_::LS;
        cx<T>* other = sl + (S_::NBUF - 1) * C * S_::LS;
        const int base = colpass ? col : row * N, stride = colpass ? N : 1;
        auto sync = [&] {
            if constexpr (P <= 32) {
                if (colpass) __syncthreads();
                else __syncwarp();
            } else {
                // a row's own P threads (whole warps) at a named barrier
                if (colpass) __syncthreads();
                else asm volatile("bar.sync %0, %1;" ::"r"(1 + c), "n"(P) : "memory");
            }
        };
        if (sp.flags & SP_LOAD) {
            const cx<T>* in = static_cast<const cx<T>*>(a.in) + base;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                using V2 = std::conditional_t<std::is_same<T, float>::value, float2, double2>;
                const V2 q = __ldcg(reinterpret_cast<const V2*>(in + L::index(t, e) * stride));
                v[e] = cx<T>{q.x, q.y};
            }
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
                    if constexpr (S_::NBUF == 2)
                        L::template forward2<true, false>(v, t, sl, other, tw_s, sync);
                    else
                        L::template forward<true, false>(v, t, sl, tw_s, sync);
                    break;
                case OP_FFT_I:
                    // a second body with conjugated twiddles is 10 % faster in
                    // complex64; in complex128 the conjugation sweeps are not
                    // on the FP64 pipe and the shorter code wins by 4 %
                    if constexpr (std::is_same<T, float>::value)
                        L::template forward2<true, true>(v, t, sl, other, tw_s, sync);
                    break;
                case OP_SCALE: {
                    const T f = (T)sh->scale;
#pragma unroll
                    for (int e = 0; e < E; ++e) v[e] = cscale(v[e], f);
                    break;
                }
                case OP_VHALF:
                    if constexpr (TAB) {
                        if (a.vtab) {
#pragma unroll
                            for (int e = 0; e < E; ++e) {
                                const double V = a.vtab[base + L::index(t, e) * stride];
                                const double an = V * (a.step_dt / (2.0 * a.hbar));
                                const double gd =
                                    a.gpe ? a.nl_coef * ((double)v[e].x * v[e].x +
                                                         (double)v[e].y * v[e].y)
                                          : 0.0;
                                if (gstate == 0) {
                                    double f = small_decay<T>(an);
                                    if (a.gpe) f *= small_decay<T>(gd);
                                    v[e] = apply_re(v[e], f);
                                } else {
                                    cx<double> f = small_phase<T>(an);
                                    if (a.gpe) f = cmul(f, small_phase<T>(gd));
                                    v[e] = apply(v[e], f);
                                }
                            }
                            break;
                        }
                    }
                    if constexpr (std::is_same<T, float>::value)
                        op_vhalf_f32<L>(v, t, vx, line_delta(lfv), a, gstate, a.nl_coef);
                    else
                        op_vhalf_sep<T, L>(v, t, vx, lfv, a, gstate, a.nl_coef);
                    break;
                case OP_KPHASE: {
                    const double ks = (sp.flags & SP_KGUARD) ? a.kscale * sh->guard : a.kscale;
                    if constexpr (std::is_same<T, float>::value)
                        op_kphase_f32<L>(v, t, ky, line_delta(lfk), (float)ks);
                    else
                        op_kphase_f64<L>(v, t, ky, cscale(lfk, ks), gstate);
                    break;
                }
                case OP_GAUGE: {
                    const int g = colpass ? 1 : 0;
                    if constexpr (TAB) {
                        if (a.atab[g]) {
                            const double* mom = a.mom[g];
#pragma unroll
                            for (int e = 0; e < E; ++e) {
                                const int i = L::index(t, e);
                                const double an = a.atab[g][base + i * stride] * mom[i] * a.gauge_dt;
                                if (gstate == 0)
                                    v[e] = apply_re(v[e], small_decay<T>(an) * a.gscale);
                                else
                                    v[e] = apply(v[e], cscale(small_phase<T>(an), a.gscale));
                            }
                            break;
                        }
                        op_gauge<T, L>(v, gauge_consts<L>(t, ang[g], gstate, a.gscale),
                                       gstate);
                    } else {
                        const cx<double>* gl = gl_s + (g * C + c) * 3;
                        op_gauge<T, L>(v, GaugeConsts{gt_s[g * nthreads + tid], gl[0], gl[1], gl[2]},
                                       gstate);
                    }
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
        if (sp.flags & SP_STORE) {
            cx<T>* out = static_cast<cx<T>*>(a.out) + base;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                using V2 = std::conditional_t<std::is_same<T, float>::value, float2, double2>;
                V2 q;
                q.x = v[e].x;
                q.y = v[e].y;
                __stcg(reinterpret_cast<V2*>(out + L::index(t, e) * stride), q);
            }
        }
        const unsigned flags = sp.flags;
        if (k + 1 < s.nseq) sp = s.seq[k + 1];  // its latency under the barrier
        if (flags & (SP_NORM | SP_GUARD)) {
            const KSum b = block_reduce(acc, sh->scratch);
            if (tid == 0) slot_store(s.slots + rank, b, (unsigned)k + 1);
        }
        if (flags & SP_SYNC) {
            target += (unsigned)ncta;
            if (!step_barrier(s.sync, target, sh)) break;
        }
        if (flags & (SP_NORM | SP_GUARD)) {
            // (a CTA overwrites its slot at the next norm only, and a barrier
            // that every reader of this one has reached lies between)
            if (tid < 32) {
                const double sum =
                    slots_sum(s.slots, ncta, (unsigned)k + 1 + sh->more_passes, sh);
                if (tid == 0) {
                    if (flags & SP_NORM) sh->scale = sqrt(sh->target_norm / sum);
                    else sh->guard = sqrt(sh->target_guard / sum);
                }
            }
            __syncthreads();
            if (sh->abort) break;
        }
    }
    __syncthreads();
    if (tid == 0) {
        if (sh->abort) {
            if (s.err) atomicExch(s.err, 1);
        } else if (rank == 0) {
            *s.scal_norm = sh->scale;
            *s.scal_guard = sh->guard;
        }
        // the last CTA of the team to leave clears the barrier for the next launch
        __threadfence();
        if (atomicAdd(s.sync + 1, 1u) == (unsigned)ncta - 1u) {
            s.sync[0] = 0u;
            for (int i = 0; i < ncta; ++i) s.slots[i] = make_double2(0.0, 0.0);  // pass 0: none
            __threadfence();
            s.sync[1] = 0u;
        }
    }
}

// A compiled stepper: the plan, its CTA limits and the kernels (void* keeps the
// launch attributes with the caller).
struct StepKernel {
    int n, ra, rb, rc, p;
    int lines;        // rows (then columns) per CTA
    size_t (*smem)(int lines);
    const void* fn[2][2];  // [tables][real time]
};
const StepKernel* find_step_kernel(int prec, int n);
const StepKernel* step_table_f32(int* count);
const StepKernel* step_table_f64(int* count);

#define GPUE_STEP(T, N, RA, RB, RC, P, C, MINB)                                              \
    StepKernel{N, RA, RB, RC, P, C, &StepShape<T, N, RA, RB, RC, P, C>::smem,                 \
               {{(const void*)&k_step2d<T, N, RA, RB, RC, P, false, false, C * P, MINB>,           \
                 (const void*)&k_step2d<T, N, RA, RB, RC, P, false, true, C * P, MINB>},           \
                {(const void*)&k_step2d<T, N, RA, RB, RC, P, true, false, C * P, MINB>,            \
                 (const void*)&k_step2d<T, N, RA, RB, RC, P, true, true, C * P, MINB>}}}

}  // namespace gpue
