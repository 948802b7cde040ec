// kernels_misc.cu -- the single-pass designs: one radix-8 stage, the
// bit-reversal unit and the full Barrett multiplication by a constant.
#include "device.cuh"

namespace gbntt {

namespace {

// One radix-8 stage exactly as the reference's NTT_R8 graph (butterfly tile
// src/kernels/ntt_r8_kernels.cc:214-404 + reduction tile :30-177): thread t of
// polynomial p reads x[i + M m] (M = n/8), forms y_k = sum_m x_m F8[m][k] in
// int32, reduces y_k with twiddle root^(i k) and writes the eight results
// (de-interleaved and 3-bit reversed, :152-154) as one 16-byte store at 8 i.
// A thread takes two adjacent i (n >= 16), so its inputs arrive as
// 4-byte pairs, its twiddles as 16-byte pairs and its outputs leave as one
// 32-byte store.  The grid's stride is a multiple of a polynomial's threads, so
// i and the eight twiddles (twice the bytes of the data) stay in registers over
// all polynomials of a thread.  Bound by issue slots and by loads in flight at
// 64 registers: 16384 x 4096 5.1 TB/s, 262144 x 256 5.4 (4.2 and 4.8 with the
// twiddles read for each polynomial; 51 registers spill, 3.9; two polynomials
// at a time 4.9 / 5.3).
constexpr int R8_THREADS = 128;
__global__ void __launch_bounds__(R8_THREADS, 8) k_r8_stage(const __grid_constant__ KArgs a, int L) {
    const int n = 1 << L, M = n >> 3;
    const int GL = L - 4;                                // log2 threads per polynomial
    const long long total = a.batch << GL, stride = (long long)gridDim.x * blockDim.x;
    const short* in = static_cast<const short*>(a.in);
    short* out = static_cast<short*>(a.out);
    const bool wide = aligned32(out);
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(idx & ((1 << GL) - 1)) * 2;      // the stride is a multiple of 2^GL
    int2 t[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int4 tt = __ldg(reinterpret_cast<const int4*>(&a.tab[k * M + i]));
        t[k][0] = make_int2(tt.x, tt.y);
        t[k][1] = make_int2(tt.z, tt.w);
    }
    grid_dep_start();
    for (; idx < total; idx += stride) {
        const long long poly = idx >> GL;
        const short* src = in + poly * n + i;
        int raw[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) raw[m] = *reinterpret_cast<const int*>(src + m * M);
        int4 v[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            int x[8], y[8], o[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) x[m] = w ? raw[m] >> 16 : (short)raw[m];
            if (a.r8_sym) {
                const int f1 = a.f8s[1], f2 = a.f8s[2], f3 = a.f8s[3];
                const int a0 = x[0] + x[4], a1 = x[1] + x[5], a2 = x[2] + x[6], a3 = x[3] + x[7];
                const int b0 = x[0] - x[4], b1 = x[1] - x[5], b2 = x[2] - x[6], b3 = x[3] - x[7];
                const int c0 = a0 + a2, c1 = a1 + a3, d0 = a0 - a2, d1 = a1 - a3;
                y[0] = c0 + c1;
                y[4] = c0 - c1;
                const int t2 = f2 * d1;
                y[2] = d0 + t2;
                y[6] = d0 - t2;
                const int e0 = b0 + f2 * b2, e1 = b0 - f2 * b2;
                const int h1 = f1 * b1 + f3 * b3, h3 = f3 * b1 + f1 * b3;
                y[1] = e0 + h1;
                y[5] = e0 - h1;
                y[3] = e1 + h3;
                y[7] = e1 - h3;
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    int acc = 0;
#pragma unroll
                    for (int m = 0; m < 8; ++m) acc += x[m] * a.f8[8 * m + k];
                    y[k] = acc;
                }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                int z = r8red(y[k], t[k][w].x, t[k][w].y, a.q);
                if (a.canonical) z = canon(z, a.q, a.canon_c);
                o[brev_c<3>(k)] = z;
            }
            v[w].x = (o[0] & 0xFFFF) | (o[1] << 16);
            v[w].y = (o[2] & 0xFFFF) | (o[3] << 16);
            v[w].z = (o[4] & 0xFFFF) | (o[5] << 16);
            v[w].w = (o[6] & 0xFFFF) | (o[7] << 16);
        }
        store_run(reinterpret_cast<int4*>(out + poly * n + 8 * i), v, wide);
    }
}

// Bit-reversal unit (src/kernels/bitreverse_kernels.cc:54-143):
// out[bitrev(i)] = in[i].  P polynomials per CTA are staged in shared memory
// with coalesced 16-byte loads, then written back in order, each thread
// reading the bit-reversed source position from shared memory.  Used for
// n < 64 and for n >= 2^13 in place (a whole polynomial per CTA); the tiled
// k_bitrev_t below, free of its bank conflicts, takes every other case.
__global__ void __launch_bounds__(256) k_bitrev(const KArgs a, int L, int P) {
    grid_dep_start();
    extern __shared__ short sb[];
    const int n = 1 << L;
    const long long poly0 = (long long)blockIdx.x * P;
    long long np = a.batch - poly0;
    if (np > P) np = P;
    const int count = (int)np << L;
    const short* src = static_cast<const short*>(a.in) + poly0 * n;
    short* dst = static_cast<short*>(a.out) + poly0 * n;
    if (n >= 8) {
        for (int j = threadIdx.x; j < count / 8; j += blockDim.x)
            reinterpret_cast<int4*>(sb)[j] = reinterpret_cast<const int4*>(src)[j];
    } else {
        for (int j = threadIdx.x; j < count; j += blockDim.x) sb[j] = src[j];
    }
    __syncthreads();
    for (int j = threadIdx.x; j < count; j += blockDim.x) {
        const int lp = j >> L, jj = j & (n - 1);
        dst[j] = sb[(lp << L) + (int)(__brev((unsigned)jj) >> (32 - L))];
    }
}

// Bit reversal of 2^L coefficients (L >= 6) as a transpose.  With
// K = min(floor(L/2), 6), m = L - 2K middle bits and the index split as (a, b, c) --
// a the top K bits, b the m middle ones, c the bottom K -- the reversed index
// is (bitrev(c), bitrev(b), bitrev(a)): for each b, the 2^K x 2^K tile
// in[a][c] lands transposed, both indices reversed, at out[bitrev(c)][bitrev(a)].
// A CTA stages whole tiles (all of a polynomial's when m = 0, so in place is
// safe) in shared memory.  Rows a and a + 2^(K-1) become neighbours, so a
// thread loads 16 bytes of both and stages the pairs of coefficients that the
// output wants in one word: an output's 16 bytes are then four words, and each
// coefficient costs half a shared-memory access a side.  The rows' padding of
// four words, the order of a thread's two 16-byte stores and the distance of a
// warp's output rows keep the accesses of K = 6 free of bank conflicts.
// 16384 x 4096: 6.8 TB/s, 262144 x 256 6.3 (4.95 and 4.96 with a word per
// coefficient and 2-way conflicts), near the 6.4-6.6 of the full Barrett unit,
// which only streams.
constexpr int BR_THREADS = 128;
template <int K>
__global__ void __launch_bounds__(BR_THREADS) k_bitrev_t(const KArgs a, int L, long long ntiles) {
    grid_dep_start();
    constexpr int S = 1 << K, TE = S * S, V = S / 8;      // V 16-byte pieces a row
    constexpr int TPC = TE >= 4096 ? 1 : 4096 / TE;      // tiles per CTA
    constexpr int PT = TE / 16, N1 = TPC * PT / BR_THREADS, N2 = 2 * N1;
    __shared__ __align__(16) int tile[TPC][S / 2][S + 4];
    const int m = L - 2 * K, tid = threadIdx.x;
    const long long t0 = (long long)blockIdx.x * TPC;
    const short* in = static_cast<const short*>(a.in);
    short* out = static_cast<short*>(a.out);
    int4 x[N1][2];
#pragma unroll
    for (int i = 0; i < N1; ++i) {
        const int e = tid + i * BR_THREADS, r = e % PT;
        const long long t = t0 + e / PT;
        const int row = r / V, c8 = (r % V) * 8;
        if (t < ntiles) {
            const short* src = in + ((t >> m) << L) + ((long long)row << (m + K)) + ((t & ((1 << m) - 1)) << K) + c8;
            x[i][0] = *reinterpret_cast<const int4*>(src);
            x[i][1] = *reinterpret_cast<const int4*>(src + ((long long)(S / 2) << (m + K)));
        }
    }
#pragma unroll
    for (int i = 0; i < N1; ++i) {
        const int e = tid + i * BR_THREADS, r = e % PT;
        const int row = r / V, c8 = (r % V) * 8;
        const int4 p = x[i][0], h = x[i][1];
        int4 lo, hi;
        lo.x = __byte_perm(p.x, h.x, 0x5410);
        lo.y = __byte_perm(p.x, h.x, 0x7632);
        lo.z = __byte_perm(p.y, h.y, 0x5410);
        lo.w = __byte_perm(p.y, h.y, 0x7632);
        hi.x = __byte_perm(p.z, h.z, 0x5410);
        hi.y = __byte_perm(p.z, h.z, 0x7632);
        hi.z = __byte_perm(p.w, h.w, 0x5410);
        hi.w = __byte_perm(p.w, h.w, 0x7632);
        int4* dst = reinterpret_cast<int4*>(&tile[e / PT][row][c8]);
        const bool second = c8 & 32;                     // the other banks first
        dst[second] = second ? hi : lo;
        dst[!second] = second ? lo : hi;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N2; ++i) {
        const int e = tid + i * BR_THREADS, tt = e / (2 * PT), r = e % (2 * PT);
        const long long t = t0 + tt;
        // rows S / 4 apart in a warp, so that their columns differ in the low bits
        const int rr = r / V, C8 = (r % V) * 8, R = ((rr & 3) << (K - 2)) | (rr >> 2);
        const int col = (int)(__brev((unsigned)R) >> (32 - K));
        if (t >= ntiles) continue;
        int w[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) w[h] = tile[tt][__brev((unsigned)(C8 + 2 * h)) >> (32 - K)][col];
        const unsigned b = (unsigned)t & ((1u << m) - 1);
        const long long br = m ? (long long)(__brev(b) >> (32 - m)) : 0;
        *reinterpret_cast<int4*>(out + ((t >> m) << L) + ((long long)R << (m + K)) + (br << K) + C8) =
            make_int4(w[0], w[1], w[2], w[3]);
    }
}

__global__ void __launch_bounds__(256) k_full_barrett(const KArgs a, long long total, int fs, int wq) {
    grid_dep_start();
    const short* in = static_cast<const short*>(a.in);
    short* out = static_cast<short*>(a.out);
    const long long nvec = total >> 3;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < nvec; j += stride) {
        const int4 w = reinterpret_cast<const int4*>(in)[j];
        int ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int lo = fb16((int)(short)(ww[h] & 0xFFFF), fs, wq, a.q);
            const int hi = fb16(ww[h] >> 16, fs, wq, a.q);
            ww[h] = (lo & 0xFFFF) | (hi << 16);
        }
        reinterpret_cast<int4*>(out)[j] = make_int4(ww[0], ww[1], ww[2], ww[3]);
    }
    for (long long j = (nvec << 3) + (long long)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += stride)
        out[j] = (short)fb16(in[j], fs, wq, a.q);
}

// grid of a grid-stride kernel: enough CTAs for the work, at most 16 per SM
int grid_for(long long work, int threads) {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 1;
    }();
    long long b = (work + threads - 1) / threads;
    const long long cap = (long long)sms * 16;
    if (b > cap) b = cap;
    return b < 1 ? 1 : (int)b;
}

}  // namespace

int bitrev_smem_bytes(int L) {
    const int n = 1 << L;
    const int P = n >= 8192 ? 1 : 8192 / n;
    return P * n * 2;
}

cudaError_t launch_r8_stage(const KArgs& a, int L, cudaStream_t s) {
    KArgs ka = a;
    void* args[] = {&ka, &L};
    // up to 32 CTAs per SM; the stride covers whole polynomials
    const int gl = L - 4;
    const unsigned unit = gl > 7 ? 1u << (gl - 7) : 1u, most = 2u * (unsigned)grid_for(a.batch << gl, 2 * R8_THREADS);
    return launch_kernel(reinterpret_cast<const void*>(&k_r8_stage), (most + unit - 1) / unit * unit, R8_THREADS, 0, args,
                         s, true, SMEM_SHARE);
}

cudaError_t launch_bitrev(const KArgs& a, int L, cudaStream_t s) {
    // buffers are 16-byte aligned (checked by the caller); beyond 2^12 a
    // polynomial's tiles spread over several CTAs, so only out of place
    if (L >= 6 && (L <= 12 || a.in != a.out)) {
        const int K = L / 2 < 6 ? L / 2 : 6;
        const long long ntiles = a.batch << (L - 2 * K);
        const int tpc = 2 * K >= 12 ? 1 : 4096 >> (2 * K);
        const unsigned grid = (unsigned)((ntiles + tpc - 1) / tpc);
        KArgs ka = a;
        int Lv = L;
        long long nt = ntiles;
        void* args[] = {&ka, &Lv, &nt};
        const void* fn = K == 3 ? reinterpret_cast<const void*>(&k_bitrev_t<3>)
                       : K == 4 ? reinterpret_cast<const void*>(&k_bitrev_t<4>)
                       : K == 5 ? reinterpret_cast<const void*>(&k_bitrev_t<5>)
                                : reinterpret_cast<const void*>(&k_bitrev_t<6>);
        return launch_kernel(fn, grid, BR_THREADS, 0, args, s, true, SMEM_SHARE);
    }
    const int n = 1 << L;
    const int P = n >= 8192 ? 1 : 8192 / n;
    const long long blocks = (a.batch + P - 1) / P;
    const int smem = P * n * 2;
    KArgs ka = a;
    int Lv = L, Pv = P;
    void* args[] = {&ka, &Lv, &Pv};
    return launch_kernel(reinterpret_cast<const void*>(&k_bitrev), (unsigned)blocks, 256, smem, args, s, true);
}

cudaError_t launch_full_barrett(const KArgs& a, long long total, int fs, int wq, cudaStream_t s) {
    KArgs ka = a;
    void* args[] = {&ka, &total, &fs, &wq};
    return launch_kernel(reinterpret_cast<const void*>(&k_full_barrett), grid_for((total + 7) / 8, 256), 256, 0, args,
                         s, true, SMEM_SHARE);
}

const void* bitrev_kernel_ptr() { return reinterpret_cast<const void*>(&k_bitrev); }

cudaError_t launch_kernel(const void* fn, unsigned grid, int threads, int smem, void** args, cudaStream_t s,
                          bool dependent, int smem_share) {
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (dependent) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (smem_share) {
        attr[n].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        attr[n++].val.sharedMemCarveout = (unsigned)smem_share;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = n ? attr : nullptr;
    cfg.numAttrs = n;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

long long large_chunk_bytes() {
    static const long long v = [] {
        const char* e = std::getenv("GBNTT_FOURSTEP_CHUNK_MB");
        const long long x = e ? std::atoll(e) : 0;
        return x >= 8 && x <= 120 ? x << 20 : 1LL << 62;
    }();
    return v;
}

}  // namespace gbntt
