// sa.cu -- best-of-restarts simulated annealing on the GPU (tessera_qa_sa_solve): the
// best-known-energy scorer for instances beyond brute force.
//
// Restates the reference's classical solver (rust/src/ising.rs:64-136, sa_run and sa_solve):
// each restart starts from a random spin pattern; sweep k runs at temperature
// t_k = t0 (t_end / t0)^(k / (max(sweeps, 2) - 1)) and visits spins 0..n-1 in order, flipping
// spin i when dE = 2 s_i (h_i + sum_j J_ij s_j) < 0 or u < exp(-dE / t_k); a run's result is
// the energy of its final pattern, and the solver keeps the lowest (the first restart on ties).
// The reference draws from rand's StdRng; here every uniform comes from a counter-based
// splitmix64 stream keyed by (seed, instance, restart, sweep, spin), so a run is reproducible
// and the CPU oracle restates it draw for draw.
//
// Layout: 8, 4 or 1 lanes per restart chain (tessera_qa_sa_solve chooses), as many CTAs per instance as it takes to fill the GPU (each
// strides over the instance's restarts); the last CTA of an instance to finish picks the winner.
// The coupling graph sits in shared memory as adjacency lists (offsets, neighbour, weight, in the
// order of the edge list); a chain's spins are a bit mask of SA_MAXN bits in registers (bit i set <->
// s_i = -1), and its local fields h_i + sum_j J_ij s_j are kept in shared memory and changed only
// where a flip changes them, the chain's lanes sharing the neighbours (one lane takes them all where
// a pair is repeated).  A visit that does not flip, the usual one once the chain has cooled, costs no
// walk over the neighbours.  With G lanes, each draws the uniform of every G-th spin and the
// temperature of every G-th sweep, and shuffles hand them round.  (Without kept fields, KEEP false, a
// field is summed at each visit.)
//
// A decision rests on the kept field and FP32 only where these can tell: u outside (1 -+ 1e-4) exp(-dE
// / t).  Of that margin __expf and the rounding of its argument take 1.2e-5 (for arguments up to 37,
// beyond which no u but 0 is as small) and the kept field at most 1e-5: fields are summed afresh every
// SA_FRESH sweeps, a task carries a bound on what rounding can do to them in between, and a sweep at a
// temperature for which that is not enough (or out of FP32's range) takes no decision this way.  All
// others are the FP64 test on the field summed there and then, neighbours in the edge list's order, so
// every decision is that test's.
//
// Bound: the latency of a visit (shuffle, field, test, a flip's walk).  8 dense n = 48 instances,
// 512 restarts x 500 sweeps: 84 ms with one thread per chain, 128 chains a CTA and the field summed
// at every visit; 20.5 ms with one CTA per 32 chains and kept fields (a warp then walks at nearly
// every visit, for whichever chain flips); 5.4 ms with 8 lanes per chain.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/tessera_qa.h"
#include "common.cuh"

namespace tq {

constexpr int SA_MAXN = 128;
constexpr int SA_WORDS = SA_MAXN / 64;
constexpr int SA_THREADS = 128;
constexpr int SA_FRESH = 64;       // sweeps between fresh sums of the kept fields
constexpr int SA_CTAS_PER_SM = 8;  // CTAs to aim at before a CTA takes more than one turn of restarts

#define SA_CK(x)                                                                                          \
    do {                                                                                                  \
        cudaError_t e_ = (x);                                                                             \
        if (e_ != cudaSuccess) throw std::runtime_error(std::string("CUDA: ") + cudaGetErrorString(e_)); \
    } while (0)

// uniform in [0, 1) from a 64-bit counter: splitmix64's finaliser (Steele, Lea and Flood 2014)
__host__ __device__ inline double sa_uniform(uint64_t seed, uint64_t inst, uint64_t restart, uint64_t sweep,
                                             uint64_t spin, uint64_t sweeps, uint64_t n) {
    uint64_t x = seed + 0x9E3779B97F4A7C15ull * ((((inst * 0x100000001B3ull + restart) * (sweeps + 1) + sweep) * n +
                                                  spin) + 1);
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    x ^= x >> 31;
    return (double)(x >> 11) * (1.0 / 9007199254740992.0);
}

struct SaTask {
    int n;
    int hoff;  // first field / spin of this instance
    int eoff;  // first edge of this instance
    int m;     // its edges (self-loops included: they enter the energy)
    int rep;   // 1: some pair of spins is coupled more than once
    double err;  // bound on what rounding makes of an energy change taken from the kept fields
};

// best chain of one CTA
struct SaBest {
    double e;
    int r;  // restart, -1 = none below infinity
    int pad;
    unsigned long long bits[SA_WORDS];
};

// lower energy first, then the lower restart; r < 0 never wins
__device__ __forceinline__ bool sa_before(const double e, const int r, const double e2, const int r2) {
    if (r < 0 || r2 < 0) return r >= 0;
    return e < e2 || (e == e2 && r < r2);
}

template <int SA_G, bool KEEP>
__global__ void __launch_bounds__(SA_THREADS) k_sa(const SaTask* tasks, const int* adj_off, const int* adj_nbr,
                                                   const double* adj_w, const double* h, const int* ei, const int* ej,
                                                   const double* ew, int restarts, int sweeps, double t0,
                                                   double t_end, unsigned long long seed, SaBest* part, int* tickets,
                                                   double* out_e, int8_t* out_s) {
    constexpr int SA_CHAINS = SA_THREADS / SA_G;
    extern __shared__ __align__(16) unsigned char smraw[];
    const SaTask tk = tasks[blockIdx.x];
    const int tid = threadIdx.x, chain = tid / SA_G, gl = tid % SA_G;
    const int n = tk.n, a0 = adj_off[tk.hoff], deg_tot = adj_off[tk.hoff + n] - a0;
    double* fld = reinterpret_cast<double*>(smraw) + chain * n;      // [n] this chain's local fields
    double* sw = reinterpret_cast<double*>(smraw) + (KEEP ? SA_CHAINS * n : 0);  // [deg_tot] weights
    double* sh = sw + deg_tot;                                       // [n] fields
    int* so = reinterpret_cast<int*>(sh + n);                        // [n + 1] offsets
    short* sn = reinterpret_cast<short*>(so + n + 1);                // [deg_tot] neighbours
    __shared__ SaBest s_best[SA_CHAINS];
    __shared__ unsigned long long s_bits[SA_CHAINS][SA_WORDS];
    __shared__ int s_last;
    for (int e = tid; e < deg_tot; e += SA_THREADS) {
        sw[e] = adj_w[a0 + e];
        sn[e] = (short)adj_nbr[a0 + e];
    }
    for (int i = tid; i < n; i += SA_THREADS) sh[i] = h[tk.hoff + i];
    for (int i = tid; i <= n; i += SA_THREADS) so[i] = adj_off[tk.hoff + i] - a0;
    __syncthreads();
    const double ratio = t_end / t0;
    const double den = (double)((sweeps < 2 ? 2 : sweeps) - 1);
    SaBest best{INFINITY, -1, 0, {}};
    // every thread of the CTA takes the same turns (a chain past the last restart runs along unseen)
    for (int r0 = blockIdx.y * SA_CHAINS; r0 < restarts; r0 += gridDim.y * SA_CHAINS) {
        const int r = r0 + chain;
        unsigned long long bits[SA_WORDS] = {};
        for (int i = gl; i < n; i += SA_G)  // random start: s_i = -1 with probability 1/2
            if (sa_uniform(seed, blockIdx.x, r, sweeps, i, sweeps, n) < 0.5) bits[i >> 6] |= 1ull << (i & 63);
#pragma unroll
        for (int o = SA_G / 2; o > 0; o >>= 1)
            for (int w = 0; w < SA_WORDS; ++w) bits[w] |= __shfl_xor_sync(0xffffffffu, bits[w], o, SA_G);
        auto field = [&](int i) {
            double f = sh[i];
            for (int e = so[i]; e < so[i + 1]; ++e) {
                const int j = sn[e];
                f += ((bits[j >> 6] >> (j & 63)) & 1ull) ? -sw[e] : sw[e];
            }
            return f;
        };
        double tl = 0.0;
        for (int k = 0; k < sweeps; ++k) {
            if (KEEP && k % SA_FRESH == 0) {
                for (int i = gl; i < n; i += SA_G) fld[i] = field(i);
                __syncwarp();
            }
            if (k % SA_G == 0) tl = t0 * pow(ratio, (double)(k + gl) / den);
            const double t = __shfl_sync(0xffffffffu, tl, k % SA_G, SA_G);
            const float it = (float)(1.0 / t);
            const bool quick = t > 1e-30 && t < 1e30 && tk.err < 1e-5 * t;
            for (int i0 = 0; i0 < n; i0 += SA_G) {
                const double ul = sa_uniform(seed, blockIdx.x, r, k, i0 + gl, sweeps, n);
                const int i1 = n - i0 < SA_G ? n - i0 : SA_G;
                for (int s = 0; s < i1; ++s) {
                    const int i = i0 + s;
                    const double u = __shfl_sync(0xffffffffu, ul, s, SA_G);
                    const bool neg = (bits[i >> 6] >> (i & 63)) & 1ull;
                    const double fk = KEEP ? fld[i] : field(i);
                    const float p = __expf((float)(neg ? fk : -fk) * 2.f * it), v = (float)u;
                    bool flip = v < p * 0.9999f;
                    if (!quick || (!flip && (!(v > p * 1.0001f) || v == 0.f))) {
                        const double f = KEEP ? field(i) : fk, de = 2.0 * (neg ? -f : f);
                        flip = de < 0.0 || u < exp(-de / t);
                    }
                    if (flip) {
                        bits[i >> 6] ^= 1ull << (i & 63);
                        const int e1 = KEEP ? so[i + 1] : 0, step = tk.rep ? 1 : SA_G;
                        for (int e = !KEEP || (tk.rep && gl) ? e1 : so[i] + gl; e < e1; e += step) {  // s_i: +2 if it was -1, else -2
                            const double w2 = 2.0 * sw[e];
                            fld[sn[e]] += neg ? w2 : -w2;
                        }
                    }
                    __syncwarp();
                }
            }
        }
        if (gl == 0)
            for (int w = 0; w < SA_WORDS; ++w) s_bits[chain][w] = bits[w];
        __syncthreads();
        if (tid < SA_CHAINS) {  // one thread a chain: E = -sum w s_i s_j - sum h s_i, in the order of the edge list
            const unsigned long long* fb = s_bits[tid];
            double en = 0.0;
            for (int e = 0; e < tk.m; ++e) {
                const int i = ei[tk.eoff + e], j = ej[tk.eoff + e];
                const int si = (fb[i >> 6] >> (i & 63)) & 1ull, sj = (fb[j >> 6] >> (j & 63)) & 1ull;
                en -= (si == sj) ? ew[tk.eoff + e] : -ew[tk.eoff + e];
            }
            for (int i = 0; i < n; ++i) en -= ((fb[i >> 6] >> (i & 63)) & 1ull) ? -sh[i] : sh[i];
            if (r0 + tid < restarts && en < best.e) {
                best.e = en;
                best.r = r0 + tid;
                for (int w = 0; w < SA_WORDS; ++w) best.bits[w] = fb[w];
            }
        }
        __syncthreads();
    }
    if (tid < SA_CHAINS) s_best[tid] = best;
    __syncthreads();
    if (tid == 0) {
        int bt = 0;
        for (int t = 1; t < SA_CHAINS; ++t)
            if (sa_before(s_best[t].e, s_best[t].r, s_best[bt].e, s_best[bt].r)) bt = t;
        part[(size_t)blockIdx.x * gridDim.y + blockIdx.y] = s_best[bt];
        __threadfence();
        s_last = atomicAdd(&tickets[blockIdx.x], 1) == (int)gridDim.y - 1;
        if (s_last) {  // the instance's last CTA: its winner over all CTAs
            __threadfence();
            const SaBest* p = part + (size_t)blockIdx.x * gridDim.y;
            int bc = 0;
            for (int c = 1; c < (int)gridDim.y; ++c)
                if (sa_before(__ldcg(&p[c].e), __ldcg(&p[c].r), __ldcg(&p[bc].e), __ldcg(&p[bc].r))) bc = c;
            s_best[0].e = __ldcg(&p[bc].e);
            for (int w = 0; w < SA_WORDS; ++w) s_best[0].bits[w] = __ldcg(&p[bc].bits[w]);
            out_e[blockIdx.x] = s_best[0].e;
        }
    }
    __syncthreads();
    if (s_last)
        for (int i = tid; i < n; i += SA_THREADS)
            out_s[tk.hoff + i] = ((s_best[0].bits[i >> 6] >> (i & 63)) & 1ull) ? -1 : 1;
}

void set_last_error(const std::string& msg);  // engine.cu: the message tessera_qa_last_error() returns

}  // namespace tq

using namespace tq;

extern "C" int tessera_qa_sa_solve(const tessera_qa_problem* problems, size_t count, size_t restarts,
                                   size_t sweeps, double t0, double t_end, uint64_t seed, int8_t* out_spins,
                                   double* out_energy) {
    char* arena = nullptr;
    cudaStream_t st = nullptr;
    auto release = [&]() {
        if (st) cudaStreamSynchronize(st);
        if (arena) device_free(arena);
        if (st) cudaStreamDestroy(st);
        arena = nullptr;
        st = nullptr;
    };
    try {
        if (!problems || count == 0 || !out_spins || !out_energy)
            throw std::invalid_argument("problems, out_spins and out_energy must be non-NULL, count >= 1");
        if (count > (1u << 20) || restarts < 1 || restarts > (1u << 20) || sweeps < 1 || sweeps > (1u << 24))
            throw std::invalid_argument("count and restarts in 1..2^20, sweeps in 1..2^24");
        if (!(t0 > 0.0) || !(t_end > 0.0) || !std::isfinite(t0) || !std::isfinite(t_end))
            throw std::invalid_argument("temperatures must be positive and finite");
        // every instance's spins are numbered from hoff; adj_off holds one offset per spin into
        // the concatenated neighbour lists, plus a final one.  The energy keeps the edge list as
        // given (self-loops included, as Ising::energy does); the dynamics skip self-loops,
        // which only add a constant.
        std::vector<SaTask> tasks(count);
        std::vector<char> seen;  // (spin, spin): coupled already
        std::vector<int> adj_off, nbr, ei, ej;
        std::vector<double> w, h, ew;
        size_t smem = 0;
        for (size_t b = 0; b < count; ++b) {
            const tessera_qa_problem& p = problems[b];
            if (p.n < 1 || p.n > (size_t)SA_MAXN || !p.h || (p.m && (!p.ei || !p.ej || !p.ew)))
                throw std::invalid_argument("instance " + std::to_string(b) + ": need 1 <= n <= " +
                                            std::to_string(SA_MAXN) + " and non-NULL arrays");
            const int n = (int)p.n;
            std::vector<std::vector<std::pair<int, double>>> adj(n);
            seen.assign(p.n * p.n, 0);
            for (int i = 0; i < n; ++i)
                if (!std::isfinite(p.h[i])) throw std::invalid_argument("non-finite field");
            SaTask t{n, (int)h.size(), (int)ei.size(), (int)p.m, 0, 0.0};
            for (size_t e = 0; e < p.m; ++e) {
                const size_t i = p.ei[e], j = p.ej[e];
                if (i >= p.n || j >= p.n || !std::isfinite(p.ew[e]))
                    throw std::invalid_argument("edge index out of range or non-finite coupling");
                ei.push_back((int)i);
                ej.push_back((int)j);
                ew.push_back(p.ew[e]);
                if (i == j) continue;
                adj[i].push_back({(int)j, p.ew[e]});
                adj[j].push_back({(int)i, p.ew[e]});
                if (seen[i * p.n + j]) t.rep = 1;
                seen[i * p.n + j] = seen[j * p.n + i] = 1;
            }
            size_t deg = 0;
            for (int i = 0; i < n; ++i) {
                h.push_back(p.h[i]);
                adj_off.push_back((int)nbr.size());
                double span = std::fabs(p.h[i]);
                for (auto& pr : adj[i]) {
                    nbr.push_back(pr.first);
                    w.push_back(pr.second);
                    span += std::fabs(pr.second);
                }
                // half an ulp of at most `span` per term: SA_FRESH sweeps in which every neighbour flips, the
                // fresh sum before them and the one the decision stands for; an energy change is twice that
                const double d = (double)adj[i].size();
                t.err = std::max(t.err, 2.0 * 0x1p-53 * span * ((SA_FRESH + 2) * d + 8.0));
                deg += adj[i].size();
            }
            tasks[b] = t;
            smem = std::max(smem, deg * (sizeof(double) + sizeof(short)) + n * sizeof(double) +
                                      (n + 1) * sizeof(int) + 64);
        }
        adj_off.push_back((int)nbr.size());
        if (smem > 200 * 1024) throw std::invalid_argument("instance graph too large for shared memory");
        size_t nmax = 0;
        for (const SaTask& t : tasks) nmax = std::max(nmax, (size_t)t.n);
        int dev = 0, sms = 0;
        SA_CK(cudaGetDevice(&dev));
        SA_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        // Lanes per chain and kept fields.  Few chains: latency rules, 8 lanes.  From 96 chains an SM on the
        // lanes compete, 4 of them: 296 dense n = 48, 256 restarts x 200 sweeps 24.3 ms against 28.7 with 8
        // and 36 with 1 (64 instances: 6.5 against 6.6, 8 instances of 32 restarts: the reverse).  From 256 an
        // SM on and at a mean degree of 8 at most, a field costs less to sum than to keep, and a chain is one
        // thread without kept fields: 296 chains of n = 48, 96 (degree 4), 128: 9.1, 16.5, 18.8 ms against 11.9,
        // 23.5, 30.5 with 4 lanes; dense n = 48 28.1 against 24.3.
        const size_t chains = count * restarts;
        const bool sum = chains >= (size_t)sms * 256 && nbr.size() <= 8 * h.size();
        const bool fits4 = smem + nmax * (SA_THREADS / 4) * sizeof(double) <= 220 * 1024;
        const int lanes = sum ? 1 : chains >= (size_t)sms * 96 && restarts >= 32 && fits4 ? 4 : 8;
        const size_t per_cta = SA_THREADS / lanes;
        if (!sum) smem += nmax * per_cta * sizeof(double);
        // CTAs per instance: one turn of restarts each, unless the batch alone fills the GPU
        const size_t turns = (restarts + per_cta - 1) / per_cta;
        const size_t share = std::max<size_t>(1, ((size_t)sms * SA_CTAS_PER_SM + count - 1) / count);
        const size_t ctas = std::min(turns, share);
        auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
        const size_t b_tasks = al(sizeof(SaTask) * count), b_off = al(sizeof(int) * adj_off.size()),
                     b_nbr = al(sizeof(int) * std::max<size_t>(nbr.size(), 1)),
                     b_w = al(sizeof(double) * std::max<size_t>(w.size(), 1)), b_h = al(sizeof(double) * h.size()),
                     b_ei = al(sizeof(int) * std::max<size_t>(ei.size(), 1)),
                     b_ew = al(sizeof(double) * std::max<size_t>(ew.size(), 1)), b_e = al(sizeof(double) * count),
                     b_s = al(h.size()), b_part = al(sizeof(SaBest) * count * ctas), b_tick = al(sizeof(int) * count);
        const size_t total = b_tasks + b_off + b_nbr + b_w + b_h + 2 * b_ei + b_ew + b_e + b_s + b_part + b_tick;
        SA_CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        SA_CK(device_alloc((void**)&arena, total, true));
        char* q = arena;
        auto take = [&](size_t bytes) { char* r = q; q += bytes; return r; };
        SaTask* d_tasks = (SaTask*)take(b_tasks);
        int* d_off = (int*)take(b_off);
        int* d_nbr = (int*)take(b_nbr);
        double* d_w = (double*)take(b_w);
        double* d_h = (double*)take(b_h);
        int* d_ei = (int*)take(b_ei);
        int* d_ej = (int*)take(b_ei);
        double* d_ew = (double*)take(b_ew);
        double* d_e = (double*)take(b_e);
        int8_t* d_s = (int8_t*)take(b_s);
        SaBest* d_part = (SaBest*)take(b_part);
        int* d_tick = (int*)take(b_tick);
        SA_CK(cudaMemsetAsync(d_tick, 0, sizeof(int) * count, st));
        auto up = [&](void* d, const void* hsrc, size_t bytes) {
            if (bytes) SA_CK(cudaMemcpyAsync(d, hsrc, bytes, cudaMemcpyHostToDevice, st));
        };
        up(d_tasks, tasks.data(), sizeof(SaTask) * count);
        up(d_off, adj_off.data(), sizeof(int) * adj_off.size());
        up(d_nbr, nbr.data(), sizeof(int) * nbr.size());
        up(d_w, w.data(), sizeof(double) * w.size());
        up(d_h, h.data(), sizeof(double) * h.size());
        up(d_ei, ei.data(), sizeof(int) * ei.size());
        up(d_ej, ej.data(), sizeof(int) * ej.size());
        up(d_ew, ew.data(), sizeof(double) * ew.size());
        auto run = [&](auto kern) {
            SA_CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            kern<<<dim3((unsigned)count, (unsigned)ctas), SA_THREADS, smem, st>>>(
                d_tasks, d_off, d_nbr, d_w, d_h, d_ei, d_ej, d_ew, (int)restarts, (int)sweeps, t0, t_end, seed, d_part,
                d_tick, d_e, d_s);
        };
        if (sum) run(k_sa<1, false>);
        else if (lanes == 4) run(k_sa<4, true>);
        else run(k_sa<8, true>);
        SA_CK(cudaGetLastError());
        std::vector<double> e(count);
        std::vector<int8_t> s(h.size());
        SA_CK(cudaMemcpyAsync(e.data(), d_e, sizeof(double) * count, cudaMemcpyDeviceToHost, st));
        SA_CK(cudaMemcpyAsync(s.data(), d_s, h.size(), cudaMemcpyDeviceToHost, st));
        SA_CK(cudaStreamSynchronize(st));
        release();
        for (size_t b = 0; b < count; ++b) out_energy[b] = e[b];
        std::copy(s.begin(), s.end(), out_spins);
        return 0;
    } catch (const std::invalid_argument& ex) {
        set_last_error(ex.what());
        release();
        return TESSERA_QA_EINVAL;
    } catch (const std::exception& ex) {
        set_last_error(ex.what());
        release();
        return TESSERA_QA_ECUDA;
    }
}
