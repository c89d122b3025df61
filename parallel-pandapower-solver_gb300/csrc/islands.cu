// islands.cu -- N-1 islanding and re-slacking on the device.
//
// Per contingency case: connected components of the live branch graph minus the case's
// outaged branches, numbered like scipy.sparse.csgraph.connected_components (ordered by
// each component's smallest bus), and the reference bus of every island: the lowest-index
// slack bus it contains, else (with reslack) its generator bus of highest priority (ties:
// lowest bus index), else none (unserved). Semantics of the reference's
// p3s/contingency/case_generator.py:355-430 (_components_after_outage, _resolve_references;
// the reference ranks generators by short-circuit impedance, this API by a caller-given
// priority, e.g. the scheduled active power).
//
// Up to 4,096 buses the labels lie in shared memory (islands_shared_kernel). Larger grids, and
// submits to a resident stream launch, take one CTA per case (persistent grid) with the labels in
// global memory. There they converge by min-label hooking with pointer jumping: every change lowers
// a label and no label drops below the smallest bus of its component, and the loop ends only when no
// edge joins two labels and every label is a root, so the fixed point labels every component with
// its smallest bus. The number of passes is bounded (checked and reported, never looped on).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "gbpf.h"
#include "gbpf_device.h"

namespace {

constexpr int NT = 256;
constexpr int NONE = 0x7fffffff;

__global__ void __launch_bounds__(NT) islands_kernel(int n, int m, const int* f, const int* t, const uint8_t* live,
                                                      int L, const int* out_ptr, const int* out_idx,
                                                      const uint8_t* is_slack, const double* prio, int reslack,
                                                      int* scratch, unsigned long long* best, int* labels,
                                                      uint8_t* served, int* ref_bus, int* n_islands, int* err) {
    int* lab = scratch + (size_t)blockIdx.x * 4 * n;
    int* id = lab + n;
    int* cslack = id + n;
    int* cgen = cslack + n;
    unsigned long long* cbest = best + (size_t)blockIdx.x * n;
    __shared__ int s_changed;
    __shared__ int s_unsettled;
    __shared__ int s_total;
    __shared__ int s_warp[NT / 32];
    const int tid = threadIdx.x;
    for (int c = blockIdx.x; c < L; c += gridDim.x) {
        const int o0 = out_ptr[c], o1 = out_ptr[c + 1];
        for (int v = tid; v < n; v += NT) lab[v] = v;
        if (tid == 0) s_unsettled = 0;
        __syncthreads();
        for (int pass = 0;; ++pass) {
            if (tid == 0) s_changed = 0;
            __syncthreads();
            for (int e = tid; e < m; e += NT) {
                if (!live[e]) continue;
                bool out = false;
                for (int q = o0; q < o1; ++q) out |= out_idx[q] == e;
                if (out) continue;
                const int a = lab[lab[f[e]]], b = lab[lab[t[e]]];
                if (a != b) {
                    const int lo = min(a, b), hi = max(a, b);
                    atomicMin(&lab[hi], lo);
                    atomicMin(&lab[f[e]], lo);
                    atomicMin(&lab[t[e]], lo);
                    s_changed = 1;
                }
            }
            __syncthreads();
            for (int v = tid; v < n; v += NT) {  // pointer jumping (bounded walk)
                const int l0 = lab[v];
                int l = l0;
                for (int k = 0; k < 64 && lab[l] != l; ++k) l = lab[l];
                if (l != l0) {
                    atomicMin(&lab[v], l);
                    s_changed = 1;
                }
            }
            __syncthreads();
            const int ch = s_changed;
            __syncthreads();
            if (!ch) break;
            if (pass > 2 * n + 64) {
                if (tid == 0) {
                    atomicCAS(err, 0, 1);
                    s_unsettled = 1;
                }
                __syncthreads();
                break;
            }
        }
        if (s_unsettled) {
            // labels that are not all roots would index the per-island words past this case's
            // islands: the case gets no islands (label -1, unserved, no reference bus) and the
            // error word, already set, is the call's only other effect
            for (int v = tid; v < n; v += NT) {
                labels[(size_t)v * L + c] = -1;
                served[(size_t)v * L + c] = 0;
                ref_bus[(size_t)v * L + c] = -1;
            }
            if (tid == 0) n_islands[c] = -1;
            __syncthreads();
            continue;
        }
        // component ids: exclusive prefix count of the roots (lab[v] == v), in bus order
        if (tid == 0) s_total = 0;
        __syncthreads();
        for (int base = 0; base < n; base += NT) {
            const int v = base + tid;
            const int r = (v < n && lab[v] == v) ? 1 : 0;
            const unsigned ball = __ballot_sync(0xffffffffu, r);
            const int lane = tid & 31, w = tid >> 5;
            if (lane == 0) s_warp[w] = __popc(ball);
            __syncthreads();
            int off = s_total;
            for (int k = 0; k < w; ++k) off += s_warp[k];
            if (r) id[v] = off + __popc(ball & ((1u << lane) - 1));
            __syncthreads();
            if (tid == 0) {
                int sum = 0;
                for (int k = 0; k < NT / 32; ++k) sum += s_warp[k];
                s_total += sum;
            }
            __syncthreads();
        }
        const int ncomp = s_total;
        for (int k = tid; k < ncomp; k += NT) {
            cslack[k] = NONE;
            cgen[k] = NONE;
            cbest[k] = 0ULL;
        }
        __syncthreads();
        // component id of every bus (roots hold theirs; read before any root is rewritten)
        for (int v = tid; v < n; v += NT) lab[v] = id[lab[v]];
        __syncthreads();
        for (int v = tid; v < n; v += NT) {
            const int k = lab[v];
            if (is_slack[v]) atomicMin(&cslack[k], v);
            if (reslack && prio[v] > 0.0) atomicMax(&cbest[k], (unsigned long long)__double_as_longlong(prio[v]));
        }
        __syncthreads();
        if (reslack)
            for (int v = tid; v < n; v += NT) {
                const int k = lab[v];
                if (prio[v] > 0.0 && (unsigned long long)__double_as_longlong(prio[v]) == cbest[k])
                    atomicMin(&cgen[k], v);
            }
        __syncthreads();
        for (int v = tid; v < n; v += NT) {
            const int k = lab[v];
            const int r = cslack[k] != NONE ? cslack[k] : (cgen[k] != NONE ? cgen[k] : -1);
            labels[(size_t)v * L + c] = k;
            served[(size_t)v * L + c] = r >= 0;
            ref_bus[(size_t)v * L + c] = r;
        }
        if (tid == 0) n_islands[c] = ncomp;
        __syncthreads();
    }
}

// The same for grids whose labels fit shared memory: 4, 2 or 1 consecutive cases a CTA, four warps
// each. A case's warps join its edges in one pass of lock-free union (a root is hooked under a smaller
// root by compare-and-swap, so a component's root is its smallest bus), flatten the trees, resolve the
// references at the roots and number the roots by ballots. What bounds it are the ~200 instructions
// and dependent label reads (25 cycles each) that a warp needs to join 32 edges; the kernel above
// makes those reads 292 cycles each in L2, over several passes with five block barriers each.
// Measured, 2,000 buses: 3,000 cases 0.43 ms there, 0.17 here; 200 cases 75 and 59 us, one case 70
// and 45 us (118 buses 15 and 9, 3,500 buses 107 and 81 us; 3,500 x 3,000 cases 0.76 and 0.40 ms).
// A CTA takes no more threads, registers or shared memory (up to 40 KB) than a 512-thread CTA of a
// stream launch: wherever one of those fits beside a resident one, so does this. (A mixed Newton CTA of
// another launch takes 6 KB without outage stamps.)
constexpr int TPC = 128;              // threads per case
constexpr int MAX_PER_THREAD = 32;    // buses of a thread, by the bits of a word
constexpr int MAX_SHARED_BUS = MAX_PER_THREAD * TPC;
constexpr int MAX_WORDS = MAX_SHARED_BUS / 32;
constexpr int SMEM_MAX = 40 * 1024;   // labels and references of a CTA's cases
constexpr int GEN = 1 << 30;          // marks a reference chosen by priority (bus below)

// Words of one case's array: at least n, and 8 mod 32, so that the writing pass, which reads four
// cases' words of eight buses at once, meets no bank twice.
__host__ __device__ constexpr int case_words(int n) { return (n + 23) / 32 * 32 + 8; }
__host__ __device__ constexpr int shared_bytes(int cases, int n) { return 2 * cases * case_words(n) * (int)sizeof(int); }
static_assert(shared_bytes(1, MAX_SHARED_BUS) <= SMEM_MAX, "one case of the largest grid must fit");

// The root of x, with path halving (without it trees of a 2,000-bus grid get so deep that the kernel
// takes twice the time of the other one). The store goes to a bus that is no root any more and puts
// an ancestor there, whatever other threads store meanwhile; labels fall along every path, so a walk
// takes at most n steps.
__device__ __forceinline__ int find_root(volatile int* lab, int x) {
    int p = lab[x];
    while (p != x) {
        const int q = lab[p];
        if (q == p) return p;
        lab[x] = q;
        x = q;
        p = lab[x];
    }
    return x;
}

template <int CASES>
__global__ void __launch_bounds__(CASES * TPC, 1024 / (CASES * TPC)) islands_shared_kernel(
    int n, int m, const int* __restrict__ f, const int* __restrict__ t, const uint8_t* __restrict__ live, int L,
    const int* __restrict__ out_ptr, const int* __restrict__ out_idx, const uint8_t* __restrict__ is_slack,
    const double* __restrict__ prio, int reslack, int* labels, uint8_t* served, int* ref_bus, int* n_islands,
    int* err) {
    extern __shared__ int s_lab[];  // labels of CASES cases, then their references
    __shared__ int s_bad[CASES];
    __shared__ unsigned s_roots[CASES][MAX_WORDS];  // which buses are roots, 32 a word
    const int w = threadIdx.x / TPC, i0 = threadIdx.x % TPC, lane = threadIdx.x & 31;
    const int stride = case_words(n), words = (n + 31) / 32;
    const long long c0 = (long long)blockIdx.x * CASES;
    const bool on = c0 + w < L;  // the last CTA's spare warps only take part in the barriers
    int* lab = s_lab + (size_t)w * stride;
    int* ref = s_lab + (size_t)(CASES + w) * stride;
    // a thread has the buses i0 + k * TPC throughout: bit k of these says what they are
    unsigned slack = 0, gen = 0, root = 0;
    if (on) {
#pragma unroll 4
        for (int k = 0; k < MAX_PER_THREAD; ++k) {
            const int v = i0 + k * TPC;
            if (v >= n) break;
            lab[v] = v;
            ref[v] = NONE;
            slack |= (is_slack[v] ? 1u : 0u) << k;
            if (reslack) gen |= (prio[v] > 0.0 ? 1u : 0u) << k;
        }
    }
    if (i0 == 0) s_bad[w] = 0;
    __syncthreads();
    if (on) {
        const int o0 = out_ptr[c0 + w], o1 = out_ptr[c0 + w + 1];
        int e = i0, na = 0, nb = 0, nl = 0;
        if (e < m) na = f[e], nb = t[e], nl = live[e];
        for (; e < m; e += TPC) {
            int a = na, b = nb;
            bool join = nl != 0;
            if (e + TPC < m) na = f[e + TPC], nb = t[e + TPC], nl = live[e + TPC];  // the next edge's, ahead
            for (int q = o0; join && q < o1; ++q) join = out_idx[q] != e;
            for (int k = 0; join; ++k) {
                a = find_root(lab, a);
                b = find_root(lab, b);
                if (a == b) break;
                const int hi = max(a, b), lo = min(a, b);
                if (atomicCAS(&lab[hi], hi, lo) == hi) break;
                if (k > n) {  // a lost swap means that another thread hooked this root: n of them at most
                    s_bad[w] = 1;
                    break;
                }
            }
        }
    }
    __syncthreads();
    if (on)
        for (int k = 0, j = i0 / 32; j < words; ++k, j += TPC / 32) {
            // every thread stores to its own bus only: a halving store could undo another's
            const int v = j * 32 + lane;
            const volatile int* vl = lab;
            int r = v;
            if (v < n) {
                for (int p; (p = vl[r]) != r;) r = p;
                *(volatile int*)&lab[v] = r;
            }
            const unsigned roots = __ballot_sync(0xffffffffu, v < n && r == v);
            if (lane == 0) s_roots[w][j] = roots;
            root |= (roots >> lane & 1u) << k;
        }
    __syncthreads();
    // slack references at the roots, then generators of islands without one
    for (unsigned s = slack; s; s &= s - 1) {
        const int v = i0 + (__ffs(s) - 1) * TPC;
        atomicMin(&ref[lab[v]], v);
    }
    __syncthreads();
    for (unsigned s = gen; s; s &= s - 1) {
        const int v = i0 + (__ffs(s) - 1) * TPC;
        int* at = &ref[lab[v]];
        int cur = *(volatile int*)at;
        if (cur < GEN) continue;  // a slack bus
        const double p = prio[v];
        for (int k = 0; k <= n; ++k) {  // a lost swap means that a better bus was set
            if (cur != NONE) {
                const double pc = prio[cur - GEN];
                if (pc > p || (pc == p && cur - GEN < v)) break;
            }
            const int was = atomicCAS(at, cur, GEN + v);
            if (was == cur) break;
            cur = was;
        }
    }
    __syncthreads();
    // a root's word becomes the complement of its island's number: the roots before it
    for (unsigned s = root; s; s &= s - 1) {
        const int v = i0 + (__ffs(s) - 1) * TPC;
        int before = __popc(s_roots[w][v / 32] & ((1u << lane) - 1));
        for (int j = 0; j < v / 32; ++j) before += __popc(s_roots[w][j]);
        lab[v] = ~before;
    }
    if (on && i0 < 32) {
        int total = 0;
        for (int j = lane; j < words; j += 32) total += __popc(s_roots[w][j]);
        total = __reduce_add_sync(0xffffffffu, total);
        if (lane == 0) {
            n_islands[c0 + w] = s_bad[w] ? -1 : total;
            if (s_bad[w]) atomicCAS(err, 0, 1);
        }
    }
    __syncthreads();
    const int q = threadIdx.x % CASES;
    if (c0 + q >= L) return;
    const int* ql = s_lab + (size_t)q * stride;
    const int* qr = s_lab + (size_t)(CASES + q) * stride;
    const bool ok = !s_bad[q];
    for (int v = threadIdx.x / CASES; v < n; v += TPC) {
        const int l = ql[v];
        const int top = l < 0 ? v : l;
        const int r = qr[top];
        const int rb = !ok || r == NONE ? -1 : (r < GEN ? r : r - GEN);
        const size_t o = (size_t)v * L + (size_t)(c0 + q);
        labels[o] = ok ? ~ql[top] : -1;
        served[o] = rb >= 0;
        ref_bus[o] = rb;
    }
}

int ifail(const std::string& m) {
    gbpf::set_error(m);
    return -1;
}

}  // namespace

cudaError_t gbpf::launch_islands(int n, int m, const int* f, const int* t, const uint8_t* live, int L,
                                 const int* out_ptr, const int* out_idx, const uint8_t* is_slack, const double* prio,
                                 int reslack, int* scratch, unsigned long long* best, int* labels, uint8_t* served,
                                 int* ref_bus, int* n_islands, int* err, int grid, cudaStream_t stream,
                                 bool beside_resident) {
    // the shared-memory kernel up to 4,096 buses, but not beside a stream launch of the same solver,
    // whose CTAs may leave a new one no room until they end
    if (n <= MAX_SHARED_BUS && !beside_resident) {
        const int cases = shared_bytes(4, n) <= SMEM_MAX ? 4 : shared_bytes(2, n) <= SMEM_MAX ? 2 : 1;
        auto* k = cases == 4 ? islands_shared_kernel<4> : cases == 2 ? islands_shared_kernel<2> : islands_shared_kernel<1>;
        k<<<(L - 1) / cases + 1, cases * TPC, shared_bytes(cases, n), stream>>>(
            n, m, f, t, live, L, out_ptr, out_idx, is_slack, prio, reslack, labels, served, ref_bus, n_islands, err);
        return cudaGetLastError();
    }
    islands_kernel<<<grid, NT, 0, stream>>>(n, m, f, t, live, L, out_ptr, out_idx, is_slack, prio, reslack, scratch,
                                            best, labels, served, ref_bus, n_islands, err);
    return cudaGetLastError();
}

cudaError_t gbpf::preload_islands() {
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, islands_kernel);
    if (!e) e = cudaFuncGetAttributes(&a, islands_shared_kernel<4>);
    if (!e) e = cudaFuncGetAttributes(&a, islands_shared_kernel<2>);
    return e ? e : cudaFuncGetAttributes(&a, islands_shared_kernel<1>);
}

extern "C" int gbpf_islands(int n, int m, const int32_t* f, const int32_t* t, const uint8_t* live, int L,
                            const int32_t* out_ptr, const int32_t* out_idx, const uint8_t* is_slack,
                            const double* gen_prio, int reslack, int32_t* labels, uint8_t* served, int32_t* ref_bus,
                            int32_t* n_islands) {
    if (n <= 0 || m < 0 || L <= 0) return ifail("gbpf_islands: invalid sizes");
    for (int e = 0; e < m; ++e)
        if (f[e] < 0 || f[e] >= n || t[e] < 0 || t[e] >= n) return ifail("gbpf_islands: branch end out of range");
    if (out_ptr[0] != 0) return ifail("gbpf_islands: outage pointers must start at 0");
    for (int c = 0; c < L; ++c)
        if (out_ptr[c + 1] < out_ptr[c]) return ifail("gbpf_islands: outage pointers must not decrease");
    const int nout = out_ptr[L];
    for (int q = 0; q < nout; ++q)
        if (out_idx[q] < 0 || out_idx[q] >= m) return ifail("gbpf_islands: outage index out of range");
    int dev = 0, nsm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int grid = std::max(1, std::min(L, 4 * nsm));
    void *df = nullptr, *dt = nullptr, *dl = nullptr, *dop = nullptr, *doi = nullptr, *ds = nullptr, *dp = nullptr,
         *dsc = nullptr, *dbest = nullptr, *dlab = nullptr, *dsv = nullptr, *dref = nullptr, *dni = nullptr,
         *derr = nullptr;
    auto al = [](void** p, size_t b) { return cudaMalloc(p, std::max<size_t>(b, 16)); };
    const size_t nl = (size_t)n * L;
    cudaError_t e = cudaSuccess;
    if (!e) e = al(&df, (size_t)m * 4);
    if (!e) e = al(&dt, (size_t)m * 4);
    if (!e) e = al(&dl, (size_t)m);
    if (!e) e = al(&dop, (size_t)(L + 1) * 4);
    if (!e) e = al(&doi, (size_t)std::max(nout, 1) * 4);
    if (!e) e = al(&ds, (size_t)n);
    if (!e) e = al(&dp, (size_t)n * 8);
    if (!e) e = al(&dsc, (size_t)grid * 4 * n * 4);
    if (!e) e = al(&dbest, (size_t)grid * n * 8);
    if (!e) e = al(&dlab, nl * 4);
    if (!e) e = al(&dsv, nl);
    if (!e) e = al(&dref, nl * 4);
    if (!e) e = al(&dni, (size_t)L * 4);
    if (!e) e = al(&derr, 16);
    if (!e && m) e = cudaMemcpy(df, f, (size_t)m * 4, cudaMemcpyHostToDevice);
    if (!e && m) e = cudaMemcpy(dt, t, (size_t)m * 4, cudaMemcpyHostToDevice);
    if (!e && m) e = cudaMemcpy(dl, live, (size_t)m, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(dop, out_ptr, (size_t)(L + 1) * 4, cudaMemcpyHostToDevice);
    if (!e && nout) e = cudaMemcpy(doi, out_idx, (size_t)nout * 4, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(ds, is_slack, (size_t)n, cudaMemcpyHostToDevice);
    if (!e && gen_prio) e = cudaMemcpy(dp, gen_prio, (size_t)n * 8, cudaMemcpyHostToDevice);
    if (!e && !gen_prio) e = cudaMemset(dp, 0, (size_t)n * 8);
    if (!e) e = cudaMemset(derr, 0, 16);
    if (!e) {
        e = gbpf::launch_islands(n, m, (const int*)df, (const int*)dt, (const uint8_t*)dl, L, (const int*)dop,
                                 (const int*)doi, (const uint8_t*)ds, (const double*)dp, reslack, (int*)dsc,
                                 (unsigned long long*)dbest, (int*)dlab, (uint8_t*)dsv, (int*)dref, (int*)dni,
                                 (int*)derr, grid, nullptr);
    }
    if (!e) e = cudaDeviceSynchronize();
    int kerr = 0;
    if (!e) e = cudaMemcpy(&kerr, derr, 4, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(labels, dlab, nl * 4, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(served, dsv, nl, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(ref_bus, dref, nl * 4, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(n_islands, dni, (size_t)L * 4, cudaMemcpyDeviceToHost);
    for (void* p : {df, dt, dl, dop, doi, ds, dp, dsc, dbest, dlab, dsv, dref, dni, derr})
        if (p) cudaFree(p);
    if (e) return ifail(std::string("gbpf_islands: ") + cudaGetErrorString(e));
    if (kerr) return ifail("gbpf_islands: label propagation did not settle");
    return 0;
}

// ---------------------------------------------------------------------------------------
// gbpf_islands_device_static: the islanding kernel on caller-owned device buffers with its
// scratch in statically allocated device memory, so a call allocates nothing (no
// cudaMalloc / cudaFree, no library routine that allocates). The scratch below is shared
// by every call on a device and keeps its last contents: the kernel initialises the label
// and per-island words it reads, and the error word is cleared before each launch. Calls
// that overlap in time on one device (other streams, other host threads) race on it.
namespace {

constexpr int STATIC_INTS = 1 << 21;  // 8 MiB: 4 n ints per CTA
constexpr int STATIC_BEST = 1 << 20;  // 8 MiB: n u64 per CTA
constexpr int STATIC_MAX_DEVICES = 64;
static_assert(GBPF_ISLANDS_STATIC_MAX_BUS <= STATIC_BEST, "one CTA must fit the static scratch");

static __device__ __align__(256) int g_static_ints[STATIC_INTS];
static __device__ __align__(256) unsigned long long g_static_best[STATIC_BEST];
static __device__ __align__(256) int g_static_err[64];

struct StaticScratch {
    int* ints = nullptr;
    unsigned long long* best = nullptr;
    int* err = nullptr;
    int nsm = 0;
    bool ready = false;
};
StaticScratch g_static[STATIC_MAX_DEVICES];
std::mutex g_static_mu;

// Validates the caller's device arrays before the islanding kernel indexes with them:
// bit 1 branch end out of range, bit 2 outage pointers not a non-decreasing 0..n_out run,
// bit 4 outage index out of range.
__global__ void islands_check_kernel(int n, int m, const int* f, const int* t, int L, const int* out_ptr,
                                     const int* out_idx, int n_out, int* err) {
    const int stride = gridDim.x * blockDim.x;
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    int bad = 0;
    for (int e = i0; e < m; e += stride)
        if (f[e] < 0 || f[e] >= n || t[e] < 0 || t[e] >= n) bad |= 1;
    for (int c = i0; c <= L; c += stride) {
        const int p = out_ptr[c];
        if (c == 0 ? p != 0 : (p < out_ptr[c - 1] || p > n_out)) bad |= 2;
        if (c == L && p != n_out) bad |= 2;
    }
    for (int q = i0; q < n_out; q += stride)
        if (out_idx[q] < 0 || out_idx[q] >= m) bad |= 4;
    if (bad) atomicOr(err, bad);
}

int static_setup(StaticScratch** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e) return ifail(std::string("gbpf_islands_device_static: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= STATIC_MAX_DEVICES) return ifail("gbpf_islands_device_static: device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_static_mu);
    StaticScratch& s = g_static[dev];
    if (!s.ready) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_ints);
        if (e) return ifail(std::string("gbpf_islands_device_static: scratch address: ") + cudaGetErrorString(e));
        s.ints = static_cast<int*>(p);
        e = cudaGetSymbolAddress(&p, g_static_best);
        if (e) return ifail(std::string("gbpf_islands_device_static: scratch address: ") + cudaGetErrorString(e));
        s.best = static_cast<unsigned long long*>(p);
        e = cudaGetSymbolAddress(&p, g_static_err);
        if (e) return ifail(std::string("gbpf_islands_device_static: scratch address: ") + cudaGetErrorString(e));
        s.err = static_cast<int*>(p);
        e = cudaDeviceGetAttribute(&s.nsm, cudaDevAttrMultiProcessorCount, dev);
        if (e) return ifail(std::string("gbpf_islands_device_static: ") + cudaGetErrorString(e));
        s.ready = true;
    }
    *out = &s;
    return 0;
}

}  // namespace

extern "C" int gbpf_islands_device_static(int n, int m, const int32_t* d_f, const int32_t* d_t,
                                          const uint8_t* d_live, int L, const int32_t* d_out_ptr,
                                          const int32_t* d_out_idx, int n_out, const uint8_t* d_is_slack,
                                          const double* d_gen_prio, int reslack, int32_t* d_labels,
                                          uint8_t* d_served, int32_t* d_ref_bus, int32_t* d_n_islands, void* stream) {
    if (n <= 0 || m < 0 || L <= 0 || n_out < 0) return ifail("gbpf_islands_device_static: invalid sizes");
    if (n > GBPF_ISLANDS_STATIC_MAX_BUS)
        return ifail("gbpf_islands_device_static: n = " + std::to_string(n) +
                     " buses exceeds the static scratch maximum of " + std::to_string(GBPF_ISLANDS_STATIC_MAX_BUS));
    if (!d_live || !d_out_ptr || !d_is_slack || !d_labels || !d_served || !d_ref_bus || !d_n_islands ||
        (m > 0 && (!d_f || !d_t)) || (n_out > 0 && !d_out_idx))
        return ifail("gbpf_islands_device_static: null device pointer");
    if (reslack && !d_gen_prio) return ifail("gbpf_islands_device_static: gen_prio is required with reslack");
    StaticScratch* s = nullptr;
    if (static_setup(&s)) return -1;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int per_cta = std::min(STATIC_INTS / (4 * n), STATIC_BEST / n);
    const int grid = std::max(1, std::min(std::min(L, 4 * s->nsm), per_cta));
    int herr = 0;
    cudaError_t e = cudaMemsetAsync(s->err, 0, sizeof(int), st);
    if (!e) {
        const int span = std::max(std::max(m, n_out), L + 1);
        const int cg = std::max(1, std::min((span + 255) / 256, 4 * s->nsm));
        islands_check_kernel<<<cg, 256, 0, st>>>(n, m, d_f, d_t, L, d_out_ptr, d_out_idx, n_out, s->err);
        e = cudaGetLastError();
    }
    if (!e) e = cudaMemcpyAsync(&herr, s->err, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaStreamSynchronize(st);
    if (e) return ifail(std::string("gbpf_islands_device_static: ") + cudaGetErrorString(e));
    if (herr & 1) return ifail("gbpf_islands_device_static: branch end out of range");
    if (herr & 2) return ifail("gbpf_islands_device_static: outage pointers must rise from 0 to n_out");
    if (herr & 4) return ifail("gbpf_islands_device_static: outage index out of range");
    e = gbpf::launch_islands(n, m, d_f, d_t, d_live, L, d_out_ptr, d_out_idx, d_is_slack, d_gen_prio, reslack, s->ints,
                             s->best, d_labels, d_served, d_ref_bus, d_n_islands, s->err, grid, st);
    if (!e) e = cudaMemcpyAsync(&herr, s->err, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaStreamSynchronize(st);
    if (e) return ifail(std::string("gbpf_islands_device_static: ") + cudaGetErrorString(e));
    if (herr) return ifail("gbpf_islands_device_static: label propagation did not settle");
    return 0;
}
