// FP64 eigenvector rotation x~ = U^T g of genotype calls on INT8 tensor cores.
//
// Calls are small integers, so U^T g needs no FP64 multiplier: each eigenvector u_i (column i
// of U) is scaled by a power of two s_i and rounded to a 56-bit integer, U_ki = s_i X_ki with
// 63.5 2^48 < max |X| <= 127 2^48, which is off by at most s_i / 2 -- 2.8e-17 of max |u_i|,
// less than the rounding of its larger elements to doubles.  The seven signed base-256 digits of X are
// its bytes after adding 128 to each (int8 digits in [-128, 127]).  Each digit product
// accumulates exactly in int32 on tcgen05 (kind::i8) and the epilogue adds the seven products
// in FP64, so the result carries a few roundings of its own size, where an FP64 GEMM carries
// those of n partial sums.
//
// Missing calls are mean-imputed without centring (src/jamma/lmm/runner_streaming.py:
// 427-434), g_j = z_j + mu_j m_j with m_j the missing mask: x~ = U^T z + mu_j U^T m.
//
// Bound by the INT8 pipe: 7 products for the calls and 7 for the masks, 28 n^2 m operations
// against 2 n^2 m on the FP64 pipe, at ~90 times its rate.
//
// Tiles: SNPs on M, digits on N.  An A tile is 128 rows: the calls of 64 SNPs and their masks,
// or the calls of 128 SNPs; a B tile is the 7 x 32 = 224 digit rows of 32 eigenvectors (digit
// t of eigenvector 32 b + e at row 224 b + 32 t + e).  All digits of an output then lie in one
// TMEM lane, 32 columns apart, and an epilogue thread of that lane adds them in registers;
// only the mask sums cross between lanes, through shared memory, on the way to the transposed
// store.  N = 224 runs at the full rate of M = 128 tiles.
// Up to n ~ 3000 a tile's products take less time than its epilogue does beside them, so eight
// warps share it (two per TMEM lane quarter, half of the eigenvectors each), the accumulator
// is released once it is read, and int32 becomes FP64 by an addition.  Paired tiles with four
// warps that released at the end -> now, 8192 SNPs: n = 1024 151 -> 115 us, n = 1940 396 -> 319,
// n = 3000 787 -> 669, n = 10 000 7.2 -> 7.2 ms; without any epilogue 78, 272, 634 us.
#include "jb_common.cuh"
#include "jb_gemm_i8.cuh"
#include "jb_rotate_i8.cuh"

namespace jb {
namespace tc {

int32_t make_map_i8(CUtensorMap* map, const void* base, int64_t rows, int64_t k, int64_t ld,
                    int box_rows);
int num_sms();

constexpr int kXDigits = 7;
constexpr int kXBN = 32 * kXDigits;   // digit rows of 32 eigenvectors
constexpr int kXStages = 4;
constexpr int kXLd = 33;              // padded row of the epilogue's output tile
constexpr int kXEpiSmem = 128 * kXLd * 8;
using XSmem = GemmSmem<kXBN, kXStages, kXEpiSmem>;

// ---------------------------------------------------------------- digit split
// Digits of four consecutive samples k..k+3 of one eigenvector (X = U f1 f2), one 32-bit word
// per digit row; rows 32 lda apart.
__device__ __forceinline__ void xsplit_store(const double (&u)[4], double f1, double f2,
                                             int8_t* __restrict__ at, int64_t lda) {
    uint32_t lo[4], hi[4];  // low and high bytes of the four samples' digits
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const long long x = __double2ll_rn(u[q] * f1 * f2);
        // bytes of X + 128 (1 + 256 + ...): digit + 128; then flip back to signed digits
        const unsigned long long b = ((unsigned long long)x + 0x0080808080808080ull) ^
                                     0x0080808080808080ull;
        lo[q] = (uint32_t)b;
        hi[q] = (uint32_t)(b >> 32);
    }
#pragma unroll
    for (int t = 0; t < kXDigits; ++t) {  // digit t: byte 6 - t
        const int by = kXDigits - 1 - t;
        const uint32_t* w = by < 4 ? lo : hi;
        const uint32_t sel = (uint32_t)((by & 3) | (((by & 3) + 4) << 4));
        const uint32_t p01 = __byte_perm(w[0], w[1], sel), p23 = __byte_perm(w[2], w[3], sel);
        *reinterpret_cast<uint32_t*>(at + 32 * t * lda) = __byte_perm(p01, p23, 0x5410);
    }
}

// One CTA per eigenvector: its scale, then its seven digit rows (bound by HBM: U read, its
// planes written).  STEPS > 0: each thread keeps its 4 STEPS elements in registers between
// the two, n <= 4 kXSplitThreads STEPS; 0: the column is read twice.  scale[i] = s_i 256^6
// (the leading digit's weight), 0 for a zero eigenvector (no digits), NaN if an element is
// not finite (every output of that row becomes NaN, as in a GEMM).
constexpr int kXSplitThreads = 512;
template <int STEPS>
__global__ void __launch_bounds__(kXSplitThreads)
    xsplit_kernel(const double* __restrict__ U, int64_t n, int64_t ldu, int8_t* __restrict__ A,
                  int64_t lda, double* __restrict__ scale) {
    const int64_t i = blockIdx.x;
    const double* __restrict__ col = U + i * ldu;
    const bool vec = (reinterpret_cast<uintptr_t>(col) & 15) == 0;
    auto load = [&](int64_t k, double (&u)[4]) {
        if (vec && k + 4 <= n) {
            const double2 a = __ldg(reinterpret_cast<const double2*>(col + k));
            const double2 b = __ldg(reinterpret_cast<const double2*>(col + k + 2));
            u[0] = a.x;
            u[1] = a.y;
            u[2] = b.x;
            u[3] = b.y;
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) u[q] = k + q < n ? __ldg(col + k + q) : 0.0;
        }
    };
    double mx = 0.0;
    bool bad = false;
    auto look = [&](const double (&u)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double a = fabs(u[q]);
            bad = bad || !(a <= 1.7976931348623157e308);
            mx = fmax(mx, a);
        }
    };
    const int64_t k0 = 4 * (int64_t)threadIdx.x, dk = 4 * (int64_t)kXSplitThreads;
    double keep[STEPS > 0 ? STEPS : 1][4];
    if (STEPS > 0) {
#pragma unroll
        for (int s = 0; s < STEPS; ++s) load(k0 + s * dk, keep[s]);
#pragma unroll
        for (int s = 0; s < STEPS; ++s) look(keep[s]);
    } else {
        for (int64_t k = k0; k < n; k += dk) {
            load(k, keep[0]);
            look(keep[0]);
        }
    }
    __shared__ double red[kXSplitThreads / 32];
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    bad = __syncthreads_or(bad);
    for (int w = 0; w < kXSplitThreads / 32; ++w) mx = fmax(mx, red[w]);
    int e = 0;  // X = U 2^e
    const bool zero = bad || !(mx > 0.0);
    if (!zero) {
        frexp(mx, &e);  // mx = f 2^e, f in [1/2, 1)
        e = 55 - e;     // mx 2^e in [2^54, 2^55)
        if (scalbn(mx, e) > 127.0 * 281474976710656.0) --e;  // the top digit holds 127 at most
    }
    if (threadIdx.x == 0)
        scale[i] = bad ? __longlong_as_double(0x7ff8000000000000ll) : (zero ? 0.0 : scalbn(1.0, 48 - e));
    // 2^e as two factors, each a normal double for every e (|e| < 1140); none without digits
    const double f1 = zero ? 0.0 : scalbn(1.0, e / 2), f2 = scalbn(1.0, e - e / 2);
    int8_t* __restrict__ rows = A + ((i / 32) * kXBN + (i % 32)) * lda;
    if (STEPS > 0) {
#pragma unroll
        for (int s = 0; s < STEPS; ++s)
            if (k0 + s * dk < lda) {
                if (bad) keep[s][0] = keep[s][1] = keep[s][2] = keep[s][3] = 0.0;
                xsplit_store(keep[s], f1, f2, rows + k0 + s * dk, lda);
            }
    } else {
        for (int64_t k = k0; k < lda; k += dk) {
            load(k, keep[0]);
            if (bad) keep[0][0] = keep[0][1] = keep[0][2] = keep[0][3] = 0.0;
            xsplit_store(keep[0], f1, f2, rows + k, lda);
        }
    }
}

// ---------------------------------------------------------------- A operand
// Block b of 64 SNPs: rows [128 b, +64) the calls (missing -> 0), rows [128 b + 64, +64) the
// masks; 16 bytes of each per thread.  SNPs and samples past the end read as call 0.
__global__ void __launch_bounds__(256) xpack_kernel(const int8_t* __restrict__ codes, int64_t ldc,
                                                    int64_t n, int64_t m, int8_t* __restrict__ A,
                                                    int64_t lda, const int* gate) {
    if (gate && !*gate) return;
    const int64_t j = blockIdx.x;
    int8_t* z = A + ((j / 64) * 128 + j % 64) * lda;
    int8_t* mk = z + 64 * lda;
    const bool vec = (reinterpret_cast<uintptr_t>(codes) & 15) == 0 && (ldc & 15) == 0;
    for (int64_t k = 16 * (int64_t)threadIdx.x; k < lda; k += 16 * (int64_t)blockDim.x) {
        uint32_t c[4] = {0u, 0u, 0u, 0u}, v[4], u[4];
        if (j < m) {
            const int8_t* row = codes + j * ldc + k;
            if (vec && k + 16 <= n) {
                const uint4 q = __ldg(reinterpret_cast<const uint4*>(row));
                c[0] = q.x;
                c[1] = q.y;
                c[2] = q.z;
                c[3] = q.w;
            } else {
                for (int q = 0; q < 16; ++q)
                    if (k + q < n) c[q >> 2] |= (uint32_t)(uint8_t)row[q] << (8 * (q & 3));
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t m3 = __vcmpeq4(c[q], 0x03030303u);
            v[q] = c[q] & ~m3;
            u[q] = m3 & 0x01010101u;
        }
        *reinterpret_cast<uint4*>(z + k) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4*>(mk + k) = make_uint4(u[0], u[1], u[2], u[3]);
    }
}

// *found = 1 if a call is missing (callers may promise that none is; the promise is checked,
// since an unmarked missing call would count as a call of 3).
__global__ void __launch_bounds__(256) xfind_missing_kernel(const int8_t* __restrict__ codes,
                                                            int64_t ldc, int64_t n, int64_t m,
                                                            int* found) {
    bool any = false;
    for (int64_t j = blockIdx.x; j < m; j += gridDim.x) {
        const int8_t* row = codes + j * ldc;  // 16-byte aligned rows (see jb_rotate_codes_f64)
        for (int64_t k = 16 * (int64_t)threadIdx.x; k < n; k += 16 * (int64_t)blockDim.x) {
            if (k + 16 <= n) {
                const uint4 q = __ldg(reinterpret_cast<const uint4*>(row + k));
                any = any || (__vcmpeq4(q.x, 0x03030303u) | __vcmpeq4(q.y, 0x03030303u) |
                              __vcmpeq4(q.z, 0x03030303u) | __vcmpeq4(q.w, 0x03030303u)) != 0u;
            } else {
                for (int64_t i = k; i < n; ++i) any = any || row[i] == 3;
            }
        }
    }
    if (__syncthreads_or(any) && threadIdx.x == 0) *found = 1;
}

// ---------------------------------------------------------------- epilogue
template <bool PAIRED>
struct XEpi {
    static constexpr int kWarps = 8;
    static constexpr int kSmem = kXEpiSmem;
    double* X;            // x~ (n x m, column-major, ld ldx)
    int64_t ldx;
    const double* scale;  // per eigenvector
    const double* mu;     // per SNP (PAIRED)
    int n, m;
    template <class Release>
    __device__ __forceinline__ void run(int mb, int nb, uint32_t taddr, int q, int lane,
                                        uint8_t* smem, Release release) const {
        double* S = reinterpret_cast<double*>(smem);  // [row][kXLd]
        constexpr int kRows = PAIRED ? 64 : 128;      // SNPs of the tile
        constexpr int kPer = kRows / kWarps;          // and of a warp's stores
        constexpr double w1 = 1.0 / 256.0;
        const int warp = (int)(threadIdx.x >> 5) - 2;
        const int row = 32 * q + lane;                // TMEM lane
        const int half = 16 * (warp >> 2);            // eigenvectors half .. half + 15 of the tile
        const int i = nb * 32 + lane;                 // eigenvector of this lane's stores
        const double sc = i < n ? __ldg(scale + i) : 0.0;
        const int64_t j0 = (int64_t)mb * kRows + warp * kPer;
        const double ml = PAIRED && lane < kPer && j0 + lane < m ? __ldg(mu + j0 + lane) : 0.0;
        // int32 to double by an addition: a conversion has a quarter of its rate
        auto dbl = [](uint32_t c) {
            return __hiloint2double(0x43300000, (int)(c ^ 0x80000000u)) - 4503601774854144.0;
        };
        // v[e] = sum_t C_t 256^-t, smallest digit first (Horner's rule from the last digit)
        static_assert(kXDigits == 7, "digits 5 and 6, 3 and 4, 1 and 2, then 0");
        double v[16];
        uint32_t c0[16], c1[16];
        const uint32_t at = taddr + (uint32_t)half;
        tmem_ld16x2(at + 5 * 32, at + 6 * 32, c0, c1);
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = fma(dbl(c1[e]), w1, dbl(c0[e]));
#pragma unroll
        for (int t = 3; t > 0; t -= 2) {
            tmem_ld16x2(at + 32 * t, at + 32 * (t + 1), c0, c1);
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = fma(fma(v[e], w1, dbl(c1[e])), w1, dbl(c0[e]));
        }
        tmem_ld16(at, c0);
        release();  // the accumulator has been read
#pragma unroll
        for (int e = 0; e < 16; ++e) S[row * kXLd + half + e] = fma(v[e], w1, dbl(c0[e]));
        epi_sync<XEpi>();
        // row by row: 32 consecutive eigenvectors of one SNP per warp store
#pragma unroll
        for (int s = 0; s < kPer; ++s) {
            const int rr = warp * kPer + s;
            double x = S[rr * kXLd + lane];
            if (PAIRED) {  // row 64 + rr: the mask sums of this SNP
                const double vm = S[(64 + rr) * kXLd + lane], u = __shfl_sync(0xffffffffu, ml, s);
                x = vm != 0.0 ? fma(u, vm, x) : x;
            }
            if (j0 + s < m && i < n) X[(j0 + s) * ldx + i] = sc * x;
        }
        epi_sync<XEpi>();  // the next tile rewrites S
    }
};

cudaError_t rotate_f64_pipeline_test_mode(int skip_loads, unsigned long long wait_limit_ns) {
    return pipeline_test_mode(skip_loads, wait_limit_ns);
}

namespace {
struct XPlanes {
    int64_t lda, rows, a_off, s_off, total;
};
XPlanes xplanes(int64_t n) {
    XPlanes L;
    L.lda = (n + 127) / 128 * 128;
    L.rows = ceil_div(n, 32) * kXBN;
    L.a_off = 0;
    L.s_off = ((L.rows * L.lda + 255) / 256) * 256;
    L.total = L.s_off + ((n * 8 + 255) / 256) * 256;
    return L;
}
// Chunk scratch: status and found words (the caller's kFirstFailure word behind them), one tile
// list per form, the packed A operand.
struct XChunk {
    int64_t status, found, tiles, tiles2, a_off, lda, total;
};
XChunk xchunk(int64_t n, int64_t m) {
    XChunk L;
    const int64_t NB = ceil_div(n, 32), MB = ceil_div(m, 64);
    auto a256 = [](int64_t x) { return (x + 255) / 256 * 256; };
    L.lda = (n + 127) / 128 * 128;
    L.status = 0;
    L.found = 4;
    L.tiles = 256;
    L.tiles2 = L.tiles + a256(MB * NB * (int64_t)sizeof(Tile));
    L.a_off = L.tiles2 + a256(ceil_div(m, 128) * NB * (int64_t)sizeof(Tile));
    L.total = L.a_off + MB * 128 * L.lda;
    return L;
}

// Tile groups: 16 SNP blocks x 9 eigenvector blocks are about one wave of CTAs, whose
// operand slices are then shared in L2.
constexpr int kXGroupM = 16, kXGroupN = 9;

template <bool PAIRED>
int32_t launch_x(const int8_t* A, int64_t a_rows, int64_t lda, const int8_t* digits,
                 const XPlanes& P, const double* scale, int64_t n, int64_t m, const double* mean,
                 double* X, int64_t ldx, Tile* tiles, int* status, const int* gate, int gate_value,
                 cudaStream_t st) {
    const int MB = (int)ceil_div(m, PAIRED ? 64 : 128), NB = (int)ceil_div(n, 32);
    CUtensorMap ta, tb;
    int32_t rc = make_map_i8(&ta, A, a_rows, n, lda, kBM);
    if (rc) return rc;
    rc = make_map_i8(&tb, digits, P.rows, n, P.lda, kXBN);
    if (rc) return rc;
    rc = launch_group_tiles(MB, NB, kXGroupM, kXGroupN, tiles, st);
    if (rc) return rc;
    auto kern = i8_gemm_kernel<kXBN, kXStages, XEpi<PAIRED>>;
    JB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, XSmem::TOTAL));
    const int64_t n_tiles = (int64_t)MB * NB;
    XEpi<PAIRED> epi{X, ldx, scale, mean, (int)n, (int)m};
    kern<<<(unsigned)(n_tiles < num_sms() ? n_tiles : num_sms()), gemm_threads<XEpi<PAIRED>>,
           XSmem::TOTAL, st>>>(
        ta, tb, tiles, (int)n_tiles, (int)ceil_div(n, kBK), epi, status, gate, gate_value);
    JB_LAUNCH_CHECK("i8_gemm_kernel<rotate f64>");
    return JB_OK;
}
}  // namespace

}  // namespace tc
}  // namespace jb

using namespace jb;
using namespace jb::tc;

extern "C" {

int64_t jb_split_f64_workspace_size(int64_t n) {
    if (n <= 0) return -1;
    return xplanes(n).total;
}

int32_t jb_split_f64_prepare(const double* U, int64_t n, int64_t ldu, void* planes,
                             int64_t planes_bytes, uintptr_t stream) {
    JB_CHECK_ARG(n > 0 && ldu >= n && U, "jb_split_f64_prepare: bad arguments");
    JB_CHECK_ARG(n < (1ll << 23), "jb_split_f64_prepare: n too large for exact int32 digit sums");
    const XPlanes P = xplanes(n);
    JB_CHECK_ARG(planes && planes_bytes >= P.total, "jb_split_f64_prepare: workspace too small");
    uint8_t* ws = static_cast<uint8_t*>(planes);
    cudaStream_t st = as_stream(stream);
    if (n % 32) {  // digit rows of the last block past the last eigenvector
        const int64_t first = (P.rows - kXBN) * P.lda;
        JB_CUDA(cudaMemsetAsync(ws + P.a_off + first, 0, (size_t)(kXBN * P.lda), st));
    }
    // P.lda is the span a CTA writes, so the register forms are chosen by it
    const int64_t step = 4 * (int64_t)kXSplitThreads;
    auto kern = P.lda <= 2 * step ? xsplit_kernel<2>
                : P.lda <= 4 * step ? xsplit_kernel<4>
                : P.lda <= 8 * step ? xsplit_kernel<8>
                : P.lda <= 12 * step ? xsplit_kernel<12>
                                     : xsplit_kernel<0>;
    kern<<<(unsigned)n, kXSplitThreads, 0, st>>>(U, n, ldu, reinterpret_cast<int8_t*>(ws + P.a_off), P.lda,
                                                 reinterpret_cast<double*>(ws + P.s_off));
    JB_LAUNCH_CHECK("xsplit_kernel");
    return JB_OK;
}

int64_t jb_rotate_codes_f64_workspace_size(int64_t n, int64_t m) {
    if (n <= 0 || m < 0) return -1;  // no SNPs: the status words
    return xchunk(n, m).total;
}

int32_t jb_rotate_codes_f64(const void* planes, int64_t n, const int8_t* codes, int64_t ld_codes,
                            int64_t m, const double* mean, int32_t has_missing, double* X,
                            int64_t ldx, void* workspace, int64_t workspace_bytes,
                            uintptr_t stream) {
    JB_CHECK_ARG(n > 0 && m >= 0 && ld_codes >= n && ldx >= n, "jb_rotate_codes_f64: bad shape");
    JB_CHECK_ARG(n < (1ll << 23) && m < (1ll << 31), "jb_rotate_codes_f64: size too large");
    if (m == 0) return JB_OK;
    JB_CHECK_ARG(planes && codes && X && mean, "jb_rotate_codes_f64: null pointer");
    const XChunk L = xchunk(n, m);
    JB_CHECK_ARG(workspace && workspace_bytes >= L.total, "jb_rotate_codes_f64: workspace too small");
    JB_CHECK_ARG(ceil_div(m, 64) * ceil_div(n, 32) < (1ll << 31), "jb_rotate_codes_f64: size too large");
    const XPlanes P = xplanes(n);
    const uint8_t* pw = static_cast<const uint8_t*>(planes);
    const int8_t* digits = reinterpret_cast<const int8_t*>(pw + P.a_off);
    const double* scale = reinterpret_cast<const double*>(pw + P.s_off);
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    int* status = reinterpret_cast<int*>(ws + L.status);
    int* found = reinterpret_cast<int*>(ws + L.found);
    int8_t* A = reinterpret_cast<int8_t*>(ws + L.a_off);
    cudaStream_t st = as_stream(stream);
    JB_CUDA(cudaMemsetAsync(ws, 0, 8, st));  // status and found
    const int* gate = nullptr;
    // without missing calls the codes are the A operand themselves (if TMA can read them);
    // should one be missing after all, the launches after it run instead
    if (!has_missing && ld_codes % 16 == 0 && (reinterpret_cast<uintptr_t>(codes) & 15) == 0) {
        gate = found;
        xfind_missing_kernel<<<(unsigned)(m < 4 * num_sms() ? m : 4 * num_sms()), 256, 0, st>>>(
            codes, ld_codes, n, m, found);
        JB_LAUNCH_CHECK("xfind_missing_kernel");
        const int32_t rc = launch_x<false>(codes, m, ld_codes, digits, P, scale, n, m, nullptr, X, ldx,
                                           reinterpret_cast<Tile*>(ws + L.tiles2), status, gate, 0, st);
        if (rc) return rc;
    }
    xpack_kernel<<<(unsigned)(ceil_div(m, 64) * 64), 256, 0, st>>>(codes, ld_codes, n, m, A, L.lda, gate);
    JB_LAUNCH_CHECK("xpack_kernel");
    return launch_x<true>(A, ceil_div(m, 64) * 128, L.lda, digits, P, scale, n, m, mean, X, ldx,
                          reinterpret_cast<Tile*>(ws + L.tiles), status, gate, 1, st);
}

}  // extern "C"
