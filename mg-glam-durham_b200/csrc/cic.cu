// Kernel (a): deterministic cloud-in-cell density, the replacement of DENSIT
// (PMP2mod_density.f90:17-301).
//
// The reference scatters eight FP64 weights per particle into the FP32 grid FI
// with `!$OMP ATOMIC` (PMP2mod_density.f90:263-279), so its summation order --
// and its last bits -- change with the thread count.  Here:
//
//   1. k_cic_count   : integer cell key of every particle; the row part of the
//                      key (J + N*K) is histogrammed with integer atomics
//                      (one per row and warp).
//   2. scan          : exclusive prefix of the N^2 row counts = row offsets.
//   3. k_cic_scatter : every particle's position is written to its row bucket
//                      (a counting sort on the row key).
//   4. k_cic_deposit : one CTA per 2 x 2 or 4 x 2 block of output rows.  It walks the
//                      records of the source rows that can reach its rows as one
//                      list, forms the reference's FP64 weights, and accumulates
//                      them in shared memory as 32.32 fixed-point integers.  Integer addition
//                      is associative, so each cell's sum -- and therefore FI --
//                      is bit-identical for any particle order, launch shape or
//                      run; the single rounding to FP32 happens at the end.
//
// Weights follow the reference exactly: D = X - INT(X) in FP64,
// w = T3*T1*(T2*WPAR) etc. (PMP2mod_density.f90:249-279), WPAR = NGRID^3/Np in
// Real*4 (line 41), FI starts at -1 (lines 47-55).
#include "mgg_internal.cuh"

#include <mutex>
#include <type_traits>

namespace mgg {

namespace {

constexpr double kFix = 4294967296.0;          // 2^32
constexpr double kUnfix = 1.0 / 4294967296.0;

__device__ __forceinline__ int cell_of(float v, int N, int32_t* flags) {
    int I = (int)v;   // 1-based, positions live in [1, N+1)
    if (!(I >= 1 && I <= N)) {
        atomicOr(flags, 1);
        I = I < 1 ? 1 : N;
    }
    return I;
}

__global__ void k_cic_count(const float* __restrict__ x, const float* __restrict__ y,
                            const float* __restrict__ z, int64_t np, int N,
                            uint32_t* __restrict__ rowcnt, uint32_t* __restrict__ slot,
                            int32_t* __restrict__ flags) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * blockDim.x) {
        (void)cell_of(__ldg(x + p), N, flags);
        const int J = cell_of(__ldg(y + p), N, flags);
        const int K = cell_of(__ldg(z + p), N, flags);
        const uint32_t r = (uint32_t)(J - 1) + (uint32_t)N * (uint32_t)(K - 1);
        // lanes with the same row (neighbouring particles usually share one) take
        // one atomic per row: the leader adds the group size, each lane its rank
        const unsigned act = __activemask();
        const unsigned grp = __match_any_sync(act, r);
        const int leader = __ffs(grp) - 1, lane = threadIdx.x & 31;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(rowcnt + r, (uint32_t)__popc(grp));
        base = __shfl_sync(act, base, leader);
        slot[p] = base + (uint32_t)__popc(grp & ((1u << lane) - 1u));
    }
}

__global__ void k_cic_scatter(const float* __restrict__ x, const float* __restrict__ y,
                              const float* __restrict__ z, int64_t np, int N,
                              const uint32_t* __restrict__ rowstart, const uint32_t* __restrict__ slot,
                              float4* __restrict__ rec) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * blockDim.x) {
        const float X = __ldg(x + p), Y = __ldg(y + p), Z = __ldg(z + p);
        int J = (int)Y, K = (int)Z;
        J = J < 1 ? 1 : (J > N ? N : J);
        K = K < 1 ? 1 : (K > N ? N : K);
        const uint32_t r = (uint32_t)(J - 1) + (uint32_t)N * (uint32_t)(K - 1);
        rec[rowstart[r] + slot[p]] = make_float4(X, Y, Z, 0.f);
    }
}

// One CTA per TY x TZ block of output rows (all N cells of each row), N = 2^lgN.
// Shared memory: TY*TZ*N fixed-point accumulators of two 32-bit words each (64 KB for
// 4 x 2 rows at N = 1024; several CTAs share an SM and hide each other's latency).
// A 64-bit add to shared memory is a compare-and-swap loop, so a value v is added
// as two 32-bit words: FIX_SPLIT, the low 20 bits and the rest, whose sums cannot
// overflow while the CTA's list is short and the particles' weight small (most
// lists; two adds that nothing waits for); FIX_CARRY, the low and high 32 bits, the
// carry taken from the low word's old value; FIX_BIG the same with the integer from
// the conversion, for particle weights from 2^17 (up to 16 particles on a 128^3 mesh,
// 8192 on 1024^3).  Below, v is at most 2^49 and the integer is read off the sum
// v + 2^52, which rounds as the conversion does; the sum is a call of its own, or the
// compiler would fuse it with v's last product, whose rounding is part of the weight.
enum FixMode { FIX_SPLIT, FIX_CARRY, FIX_BIG };
constexpr float kBigWpar = 131072.0f;   // v <= 2^32 weight, far enough below the 2^52 that the sum needs
template <FixMode MODE>
__device__ __forceinline__ void fix_add(uint32_t* lo, uint32_t* hi, int cell, double v) {
    const unsigned long long b = MODE == FIX_BIG ? __double2ull_rn(v)
                                                 : (unsigned long long)__double_as_longlong(__dadd_rn(v, 4503599627370496.0));
    const uint32_t l = (uint32_t)b, hw = (uint32_t)(b >> 32);
    if (MODE == FIX_SPLIT) {
        atomicAdd(lo + cell, l & 0xfffffu);
        atomicAdd(hi + cell, __funnelshift_r(l, hw, 20));   // the exponent bits of v + 2^52 shift out
        return;
    }
    const uint32_t old = atomicAdd(lo + cell, l);
    const uint32_t h = (MODE == FIX_BIG ? hw : hw & 0xfffffu) + (old > ~l ? 1u : 0u);
    if (h) atomicAdd(hi + cell, h);
}

// The source rows that reach the block are rows j0-1 .. j0+TY-1 of the planes k0-1 ..
// k0+TZ-1; a plane's rows sit side by side in rec (two runs where j0-1 wraps), so
// the block walks TZ+1 (or twice as many) runs as one list and no thread idles on a
// short row.
template <int TY, int TZ, int NT>
__global__ void __launch_bounds__(NT) k_cic_deposit(const float4* __restrict__ rec,
                                                             const uint32_t* __restrict__ rowstart, int N, int lgN,
                                                             float wpar, float* __restrict__ fi) {
    extern __shared__ uint32_t acc[];
    constexpr int MAXRUN = 2 * (TZ + 1);
    __shared__ uint32_t run_end[MAXRUN], run_off[MAXRUN];   // ends in the list; record - list position
    const int j0 = blockIdx.x * TY, k0 = blockIdx.y * TZ;
    const int nacc = (TY * TZ) << lgN;
    uint32_t* lo = acc;
    uint32_t* hi = acc + nacc;
    for (int e = threadIdx.x; e < 2 * nacc; e += NT) acc[e] = 0u;
    const bool wrap = j0 == 0;
    const int nrun = wrap ? MAXRUN : TZ + 1;
    if (threadIdx.x < 32) {
        const int r = threadIdx.x;
        uint32_t beg = 0, len = 0;
        if (r < nrun) {
            const int pl = wrap ? r >> 1 : r;
            const int sk = (k0 - 1 + pl) & (N - 1);
            const int first = wrap ? (r & 1 ? 0 : N - 1) : j0 - 1, last = wrap && !(r & 1) ? N - 1 : j0 + TY - 1;
            beg = __ldg(rowstart + ((uint32_t)first + ((uint32_t)sk << lgN)));
            len = __ldg(rowstart + ((uint32_t)last + ((uint32_t)sk << lgN) + 1)) - beg;
        }
        uint32_t end = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
            if (r >= o) end += y;
        }
        if (r < nrun) {
            run_end[r] = end;
            run_off[r] = beg - (end - len);
        }
    }
    __syncthreads();
    const double W = (double)wpar * kFix;   // a power of two: the weights' bits are the unscaled ones
    const uint32_t total = run_end[nrun - 1];
    const bool split = total < 4096u && wpar * (float)total < 1048576.0f;
    auto deposit = [&](auto mode) {
      constexpr FixMode MODE = decltype(mode)::value;
      for (uint32_t q = threadIdx.x; q < total; q += NT) {
        int run = 0;
        while (q >= run_end[run]) ++run;
        const float4 r = __ldg(rec + (q + run_off[run]));
        int I = (int)r.x;
        I = I < 1 ? 1 : (I > N ? N : I);
        int Jc = (int)r.y, Kc = (int)r.z;
        const double D1 = (double)r.x - (double)(float)I, D2 = (double)r.y - (double)(float)Jc,
                     D3 = (double)r.z - (double)(float)Kc;
        const double T1 = 1.0 - D1, T2 = 1.0 - D2, T3 = 1.0 - D3;
        const double T2W = T2 * W, D2W = D2 * W;
        const int i0 = I - 1, i1 = (I == N) ? 0 : I;
        // the bucket's row (a position clamped by the count sits in the clamped row)
        Jc = Jc < 1 ? 1 : (Jc > N ? N : Jc);
        Kc = Kc < 1 ? 1 : (Kc > N ? N : Kc);
        // target rows inside the block
        const int jj0 = Jc - 1 - j0, jj1 = (Jc == N ? 0 : Jc) - j0;
        const int kk0 = Kc - 1 - k0, kk1 = (Kc == N ? 0 : Kc) - k0;
        const bool vj0 = (unsigned)jj0 < (unsigned)TY, vj1 = (unsigned)jj1 < (unsigned)TY;
        if ((unsigned)kk0 < (unsigned)TZ) {
            const double a = T3 * T1, b = T3 * D1;
            if (vj0) {
                const int c = (kk0 * TY + jj0) << lgN;
                fix_add<MODE>(lo, hi, c + i0, a * T2W);
                fix_add<MODE>(lo, hi, c + i1, b * T2W);
            }
            if (vj1) {
                const int c = (kk0 * TY + jj1) << lgN;
                fix_add<MODE>(lo, hi, c + i0, a * D2W);
                fix_add<MODE>(lo, hi, c + i1, b * D2W);
            }
        }
        if ((unsigned)kk1 < (unsigned)TZ) {
            const double a = D3 * T1, b = D3 * D1;
            if (vj0) {
                const int c = (kk1 * TY + jj0) << lgN;
                fix_add<MODE>(lo, hi, c + i0, a * T2W);
                fix_add<MODE>(lo, hi, c + i1, b * T2W);
            }
            if (vj1) {
                const int c = (kk1 * TY + jj1) << lgN;
                fix_add<MODE>(lo, hi, c + i0, a * D2W);
                fix_add<MODE>(lo, hi, c + i1, b * D2W);
            }
        }
      }
    };
    if (split) deposit(std::integral_constant<FixMode, FIX_SPLIT>{});
    else if (wpar < kBigWpar) deposit(std::integral_constant<FixMode, FIX_CARRY>{});
    else deposit(std::integral_constant<FixMode, FIX_BIG>{});
    __syncthreads();
    const int64_t NN = (int64_t)N;
    for (int e = threadIdx.x; e < nacc; e += NT) {
        const int i = e & (N - 1), rowl = e >> lgN;
        const int jj = rowl % TY, kk = rowl / TY;
        const double v = (double)(((unsigned long long)hi[e] << (split ? 20 : 32)) + lo[e]) * kUnfix - 1.0;
        fi[(int64_t)i + NN * ((int64_t)(j0 + jj) + NN * (int64_t)(k0 + kk))] = (float)v;
    }
}

int ilog2i(int n) {
    int l = 0;
    while ((1 << l) < n) ++l;
    return l;
}

// deposit launch for an N^3 grid (N a power of two, 16 <= N <= 1024)
void launch_deposit(const float4* rec, const uint32_t* rowstart, int N, float wpar, float* fi, cudaStream_t s) {
    // 4 x 2 rows a CTA visit a record 1.9 times on average, 2 x 2 rows 2.25 times, but small meshes need
    // the CTAs: 2.95 -> 2.87 ms at 1024^3 (512^3 particles), 0.439 -> 0.420 at 512^3, equal at 256^3
    if (N >= 512) {
        k_cic_deposit<4, 2, 512><<<dim3(N / 4, N / 2), 512, (size_t)8 * N * 8, s>>>(rec, rowstart, N, ilog2i(N), wpar, fi);
    } else {
        k_cic_deposit<2, 2, 256><<<dim3(N / 2, N / 2), 256, (size_t)4 * N * 8, s>>>(rec, rowstart, N, ilog2i(N), wpar, fi);
    }
}

}  // namespace

void cic_alloc(Ctx& c) {
    const int64_t rows = (int64_t)c.N * c.N;
    MGG_CUDA(cudaFuncSetAttribute(k_cic_deposit<4, 2, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    MGG_CUDA(cudaMalloc(&c.cic_rowcnt, sizeof(uint32_t) * (rows + 1)));
    MGG_CUDA(cudaMalloc(&c.cic_rowstart, sizeof(uint32_t) * (rows + 1)));
    MGG_CUDA(cudaMalloc(&c.cic_slot, sizeof(uint32_t) * c.np));
    MGG_CUDA(cudaMalloc(&c.cic_rec, sizeof(float4) * c.np));
}

void cic_grid(Ctx& c, const float* x, const float* y, const float* z, int N, float* out) {
    const int64_t rows = (int64_t)N * N;
    c.cic_last_n = N;
    const int threads = 256;
    const int blocks = (int)std::min<int64_t>(div_up(c.np, threads), 148 * 16);
    MGG_CUDA(cudaMemsetAsync(c.cic_rowcnt, 0, sizeof(uint32_t) * (rows + 1), c.stream));
    {
        ProfScope ps(c, K_CIC_COUNT, 16.0 * c.np);
        k_cic_count<<<blocks, threads, 0, c.stream>>>(x, y, z, c.np, N, c.cic_rowcnt, c.cic_slot, c.d_flags);
        MGG_CHECK_LAUNCH();
    }
    {
        ProfScope ps(c, K_SCAN, 8.0 * (double)(rows + 1));
        scan_exclusive(c.cic_rowcnt, c.cic_rowstart, c.scan_tmp, rows + 1, c.stream);
    }
    {
        ProfScope ps(c, K_CIC_SCATTER, 32.0 * c.np);
        k_cic_scatter<<<blocks, threads, 0, c.stream>>>(x, y, z, c.np, N, c.cic_rowstart, c.cic_slot, c.cic_rec);
        MGG_CHECK_LAUNCH();
    }
    {
        ProfScope ps(c, K_CIC_DEPOSIT, 12.0 * c.np + 4.0 * (double)N * N * N);
        launch_deposit(c.cic_rec, c.cic_rowstart, N, (float)((double)N * N * N / (double)(float)c.np), out, c.stream);
        MGG_CHECK_LAUNCH();
    }
}

namespace {

// Per-cell counts recounted from the row buckets: block r walks bucket r and
// counts each record into cell (INT(X), r), so a record placed in the wrong
// bucket would land in the wrong cell.
__global__ void k_cic_cellcount(const float4* __restrict__ rec, const uint32_t* __restrict__ rowstart, int N,
                                uint32_t* __restrict__ cellcnt) {
    const uint32_t row = blockIdx.x + (uint32_t)N * blockIdx.y;
    const uint32_t beg = rowstart[row], end = rowstart[row + 1];
    for (uint32_t q = beg + threadIdx.x; q < end; q += blockDim.x) {
        int I = (int)rec[q].x;
        I = I < 1 ? 1 : (I > N ? N : I);
        atomicAdd(cellcnt + (size_t)row * N + (I - 1), 1u);
    }
}

}  // namespace

void cic_keys(Ctx& c, uint32_t* rowcnt, uint32_t* rowstart, uint32_t* cellcnt) {
    const int N = c.N;
    if (c.cic_last_n != N) throw Error{MGG_ERR_STATE, "cic_keys: no density on the NGRID mesh since the last analysis call"};
    const int64_t rows = (int64_t)N * N;
    if (rowcnt) MGG_CUDA(cudaMemcpyAsync(rowcnt, c.cic_rowcnt, sizeof(uint32_t) * rows, cudaMemcpyDeviceToHost, c.stream));
    if (rowstart)
        MGG_CUDA(cudaMemcpyAsync(rowstart, c.cic_rowstart, sizeof(uint32_t) * (rows + 1), cudaMemcpyDeviceToHost, c.stream));
    if (cellcnt) {
        uint32_t* d = nullptr;
        const size_t b = sizeof(uint32_t) * (size_t)c.ncell;
        if (cudaMalloc(&d, b) != cudaSuccess) {
            cudaGetLastError();
            throw Error{MGG_ERR_NOMEM, "cic_keys: no device memory for the cell counts"};
        }
        try {
            MGG_CUDA(cudaMemsetAsync(d, 0, b, c.stream));
            k_cic_cellcount<<<dim3(N, N), 128, 0, c.stream>>>(c.cic_rec, c.cic_rowstart, N, d);
            MGG_CHECK_LAUNCH();
            MGG_CUDA(cudaMemcpyAsync(cellcnt, d, b, cudaMemcpyDeviceToHost, c.stream));
            MGG_CUDA(cudaStreamSynchronize(c.stream));
        } catch (...) {
            cudaStreamSynchronize(c.stream);
            cudaFree(d);
            throw;
        }
        MGG_CUDA(cudaFree(d));
    }
    MGG_CUDA(cudaStreamSynchronize(c.stream));
}

void cic_density(Ctx& c) {
    if (!c.have_particles) throw Error{MGG_ERR_STATE, "density: no particles uploaded"};
    BucketScope bs(c, MGG_T_DENSITY);
    cic_grid(c, c.x, c.y, c.z, c.N, c.fi);
}

// ---------------------------------------------------------------------------
// Density without allocation.  Some callers cannot call cudaMalloc: a host
// that owns all device memory through its own pool or arena (and forbids
// other allocations in its process), or code that runs where an allocation
// could synchronise the device at the wrong moment.  This variant of the CIC
// pipeline above takes the caller's device arrays and keeps its bucketing
// scratch (row counts, row offsets, per-particle slots and records, the range
// flag) in one file-scope device array of fixed size, kNoAllocBytes (about
// 40.5 MiB), which every GPU that loads this library holds until the process
// exits.  Limits: NGRID a power of two in [16, 256] and at most 2^21
// particles.  The first call on each device looks up the array's device
// address (cudaGetSymbolAddress) with that device current and keeps it for
// the life of the process, so a cudaDeviceReset between calls is not
// supported.  The stream must belong to the current device.  Every call waits
// for its own range flag on the host, so no call can be made while its stream
// is being captured into a CUDA graph (such a call is refused before it
// queues any work).  All calls share the one array and it keeps the last
// call's contents: the row counts and the flag are cleared on every call, and
// calls that overlap on the GPU (other threads or streams) race.
// ---------------------------------------------------------------------------
namespace {

constexpr int kNoAllocMaxNgrid = 256;
constexpr int64_t kNoAllocMaxParticles = int64_t(1) << 21;
constexpr size_t kNoAllocRows = (size_t)kNoAllocMaxNgrid * kNoAllocMaxNgrid + 1;
constexpr size_t align256(size_t b) { return (b + 255) / 256 * 256; }
// the range flag sits before the row counts, so that one clear covers both; then the scan's block sums
constexpr size_t kNaOffFlags = 0, kNaOffRowcnt = 256;
constexpr size_t kNaOffRowstart = kNaOffRowcnt + align256(sizeof(uint32_t) * kNoAllocRows);
constexpr size_t kNaOffSlot = kNaOffRowstart + align256(sizeof(uint32_t) * kNoAllocRows);
constexpr size_t kNaOffRec = kNaOffSlot + align256(sizeof(uint32_t) * kNoAllocMaxParticles);
constexpr size_t kNaOffSums = kNaOffRec + align256(sizeof(float4) * kNoAllocMaxParticles);
constexpr size_t kNoAllocBytes = kNaOffSums + 256;   // 9 block sums at NGRID = 256

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kMaxDevices] = {};

}  // namespace

void density_noalloc(const float* x, const float* y, const float* z, int64_t np, int ngrid, float* fi,
                     cudaStream_t stream) {
    if (!x || !y || !z || !fi) throw Error{MGG_ERR_ARG, "density_noalloc: null pointer"};
    if (ngrid < 16 || ngrid > kNoAllocMaxNgrid || (ngrid & (ngrid - 1)) != 0)
        throw Error{MGG_ERR_ARG, "density_noalloc: NGRID must be a power of two in [16, 256]"};
    if (np < 1 || np > kNoAllocMaxParticles)
        throw Error{MGG_ERR_ARG, "density_noalloc: particle count must be in [1, 2097152]"};
    int dev = 0;
    MGG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) throw Error{MGG_ERR_ARG, "density_noalloc: device index out of range"};
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    MGG_CUDA(cudaStreamIsCapturing(stream, &cap));
    if (cap != cudaStreamCaptureStatusNone)
        throw Error{MGG_ERR_STATE, "density_noalloc: the stream is being captured (the call waits for its result)"};
    int sdev = dev;
    MGG_CUDA(cudaStreamGetDevice(stream, &sdev));
    if (sdev != dev) throw Error{MGG_ERR_ARG, "density_noalloc: the stream belongs to another device"};
    unsigned char* base = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {   // once per device, with that device current
            void* p = nullptr;
            MGG_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
            g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
        }
        base = g_noalloc_ptr[dev];
    }
    uint32_t* rowcnt = reinterpret_cast<uint32_t*>(base + kNaOffRowcnt);
    uint32_t* rowstart = reinterpret_cast<uint32_t*>(base + kNaOffRowstart);
    uint32_t* slot = reinterpret_cast<uint32_t*>(base + kNaOffSlot);
    float4* rec = reinterpret_cast<float4*>(base + kNaOffRec);
    int32_t* flags = reinterpret_cast<int32_t*>(base + kNaOffFlags);
    const int N = ngrid;
    const int64_t rows = (int64_t)N * N;
    const int threads = 256;
    const int blocks = (int)std::min<int64_t>(div_up(np, threads), 148 * 16);
    MGG_CUDA(cudaMemsetAsync(base, 0, kNaOffRowcnt + sizeof(uint32_t) * (rows + 1), stream));   // flag and counts
    k_cic_count<<<blocks, threads, 0, stream>>>(x, y, z, np, N, rowcnt, slot, flags);
    MGG_CHECK_LAUNCH();
    scan_exclusive(rowcnt, rowstart, reinterpret_cast<uint32_t*>(base + kNaOffSums), rows + 1, stream);
    k_cic_scatter<<<blocks, threads, 0, stream>>>(x, y, z, np, N, rowstart, slot, rec);
    MGG_CHECK_LAUNCH();
    launch_deposit(rec, rowstart, N, (float)((double)N * N * N / (double)(float)np), fi, stream);
    MGG_CHECK_LAUNCH();
    int32_t h = 0;
    MGG_CUDA(cudaMemcpyAsync(&h, flags, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    MGG_CUDA(cudaStreamSynchronize(stream));
    if (h) throw Error{MGG_ERR_NUMERIC, "density_noalloc: particle position outside [1, NGRID+1) (clamped)"};
}

}  // namespace mgg
