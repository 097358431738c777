// Pack / layout kernels.  All integer work, bit-exact with the reference's
// PyTorch packers (src/nanoquant/kernel/utils.py in the reference project):
//
//   rows layout    int32 [rows, ceil(cols/32)], bit order lsb_first or half2
//   marlin layout  int32 [in/16, out/2], one word = the B fragments of one lane
//   tile layout    the runtime layout of the GEMV kernel here, see nq_rows_to_tiles
//
// Each thread produces whole output words so that stores are coalesced; the
// kernels are bound by the bytes they read and write.
#include "nq_common.cuh"

namespace nq {

constexpr int kPackThreads = 256;

static inline unsigned grid_for(int64_t n, int threads) {
    int64_t g = (n + threads - 1) / threads;
    const int64_t cap = 148LL * 64;  // grid-stride beyond this
    return static_cast<unsigned>(g < 1 ? 1 : (g > cap ? cap : g));
}

// Launches with programmatic stream serialization and no early trigger: packing is a run of such calls, and the blocks of the
// next one are set up while this one's last blocks finish (pack, tiles and unpack of 12288 x 2432 in a stream: 33.7 -> 28.4
// us).  The kernels touch memory only behind enter().  They do NOT let a successor in early: the linears load their weight
// tiles ahead of their own dependency wait, so the tiles have to be complete by then.
template <typename... P, typename... A>
static int launch(void (*kernel)(P...), unsigned grid, unsigned threads, nq_stream_t stream, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.stream = as_stream(stream);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    NQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
    return NQ_OK;
}
__device__ __forceinline__ void enter() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// sign bits of four int8 values held in one register -> 4-bit field (byte b -> bit b)
__device__ __forceinline__ uint32_t sign_nibble(uint32_t v) {
    uint32_t x = (v >> 7) & 0x01010101u;
    return (x * 0x01020408u) >> 24;  // gathers bits 0,8,16,24 into bits 0..3
}

// 4-bit field -> bit b placed at position 8*b
__device__ __forceinline__ uint32_t spread_nibble(uint32_t n) {
    return ((n & 0xFu) * 0x00204081u) & 0x01010101u;
}

// ---------------------------------------------------------------------------
// rows layout
// ---------------------------------------------------------------------------
// Matrices of any width at any address.  The rows are one run of bytes, in which a word starts at any byte, so a thread
// that fetches its own 32 bytes can only do so byte by byte.  Here a warp takes 64 consecutive words: the up to 129 aligned
// 16-byte pieces that cover them come in with contiguous loads, each piece leaves its 16 sign bits in shared memory, and a
// word is 32 bits of that string.  The instructions bound it, hence one division per 2 KB and offsets inside a step in 32
// bits (they are small: sums modulo 2^32 will do).  12291 x 2435: 8.7 us (29.7 with byte loads).
constexpr int kAnyThreads = 128;      // small blocks: a matrix of a few hundred KB is a few hundred warps

// a / b for a >= 0, b > 0, in 32 bits where that will do (the same branch in the whole warp)
__device__ __forceinline__ int64_t quotient(int64_t a, int64_t b) {
    return ((a | b) >> 32) == 0 ? (int64_t)((uint32_t)a / (uint32_t)b) : a / b;
}
// Element `d` behind element `col` of a row of `n` elements: rows crossed, and the column in its row; 0 <= d <= 2048
__device__ __forceinline__ uint32_t advance(int64_t& col, int d, int64_t n) {
    col += d;
    if (n >= 2048) {                            // col < n before: one row at most
        if (col < n) return 0;
        col -= n;
        return 1;
    }
    const uint32_t q = (uint32_t)col / (uint32_t)n;
    col -= (int64_t)(q * (uint32_t)n);
    return q;
}
// signs of 16 int8 values -> 16 bits.  The products put bits 7, 15, 23, 31 of a word at 28..31.
__device__ __forceinline__ uint32_t sign_bits16(const uint4& v) {
    auto top4 = [](uint32_t x) { return (x & 0x80808080u) * 0x00204081u; };
    uint32_t h = top4(v.w) >> 28;
    h = __funnelshift_l(top4(v.z), h, 4);
    h = __funnelshift_l(top4(v.y), h, 4);
    return __funnelshift_l(top4(v.x), h, 4);
}
// 16 bits -> int8 +1 (0) / -1 (1): bit b of a nibble goes to bit 8b + 7, whose byte is filled with it, lowest bit set
__device__ __forceinline__ uint4 signs_of16(uint32_t h) {
    auto four = [](uint32_t product) {
        uint32_t fill;     // selector values 8..11: the sign of byte 0..3, repeated (__byte_perm drops that bit)
        asm("prmt.b32 %0, %1, 0, 0xBA98;" : "=r"(fill) : "r"(product));
        return fill | 0x01010101u;
    };
    const uint32_t g = h >> 8;
    return make_uint4(four((h & 0x0Fu) * 0x10204080u), four((h & 0xF0u) * 0x01020408u), four((g & 0x0Fu) * 0x10204080u),
                      four((g & 0xF0u) * 0x01020408u));
}

__global__ void __launch_bounds__(kAnyThreads) pack_rows_kernel(const int8_t* __restrict__ w, uint32_t* __restrict__ out,
                                                                int64_t rows, int64_t cols, int64_t words, int order) {
    enter();
    __shared__ uint32_t signs[kAnyThreads / 32][66];     // 16 bits per piece, piece 2i in the low half of word i
    const int lane = threadIdx.x & 31;
    uint32_t* const mine = signs[threadIdx.x >> 5];
    const int64_t total = rows * words, bytes = rows * cols, step = (int64_t)gridDim.x * (kAnyThreads / 32) * 64;
    const uint32_t tail = (uint32_t)(cols - 32 * (words - 1));                   // columns in a row's last word
    for (int64_t base = ((int64_t)blockIdx.x * (kAnyThreads / 32) + (threadIdx.x >> 5)) * 64; base < total; base += step) {
        const int64_t r0 = quotient(base, words), wi0 = base - r0 * words, b0 = r0 * cols + 32 * wi0;
        const int mis = (int)((reinterpret_cast<uintptr_t>(w) + (uintptr_t)b0) & 15);
        // pieces [lo, hi) lie inside the matrix; the one before and the one after may do so in part
        const int lo = b0 < mis ? 1 : 0, hi = bytes - b0 + mis < 129 * 16 ? (int)(bytes - b0 + mis) >> 4 : 129;
        const int8_t* const from = w + (b0 - mis);
        uint4 v[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const int p = 32 * k + lane;
            v[k] = p >= lo && p < hi ? __ldcs(reinterpret_cast<const uint4*>(from) + p) : make_uint4(0u, 0u, 0u, 0u);
        }
        uint16_t* const piece = reinterpret_cast<uint16_t*>(mine);
        __syncwarp();                                                            // the previous step's string has been read
#pragma unroll
        for (int k = 0; k < 5; ++k)
            if (k < 4 || lane < 4) piece[32 * k + lane] = (uint16_t)sign_bits16(v[k]);
        if (lo > 0 || hi < 129) {                                                // (the whole warp) an end of the matrix
            __syncwarp();
            const int p = lane == 0 ? 0 : hi;
            if ((lane == 0 && lo > 0) || (lane == 1 && hi < 129)) {
                uint32_t h = 0;
                const int64_t f = b0 - mis + 16 * p;
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (f + e >= 0 && f + e < bytes) h |= (uint32_t)(w[f + e] < 0) << e;
                piece[p] = (uint16_t)h;
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            int64_t wi = wi0;
            const uint32_t dr = advance(wi, 32 * k + lane, words);
            if (base + 32 * k + lane < total) {
                const uint32_t at = (uint32_t)mis + dr * (uint32_t)cols + 32u * (uint32_t)(wi - wi0);   // below 16 + 2048
                uint32_t v32 = __funnelshift_r(mine[at >> 5], mine[(at >> 5) + 1], at & 31);
                if (wi == words - 1) v32 &= 0xFFFFFFFFu >> (32 - tail);          // padding stays +1 (bit 0)
                out[base + 32 * k + lane] = convert_order(v32, NQ_LSB_FIRST, order);
            }
        }
    }
}

// The way back: a warp writes 32 * P of the aligned 16-byte pieces of the run of bytes.  A lane gathers the 16 bits of a
// piece from the one or two words that hold them, the words of all its pieces in flight together; pieces that span rows, or
// an end of the matrix, go bit run by bit run.  12291 x 2435: 12.5 us (172 with byte stores).
template <int P>
__global__ void __launch_bounds__(kAnyThreads) unpack_rows_kernel(const uint32_t* __restrict__ packed, int8_t* __restrict__ w,
                                                                  int64_t rows, int64_t cols, int64_t words, int order) {
    enter();
    const int lane = threadIdx.x & 31, mis = (int)(reinterpret_cast<uintptr_t>(w) & 15);
    const int64_t bytes = rows * cols, pieces = (bytes + mis + 15) / 16, step = (int64_t)gridDim.x * (kAnyThreads * P);
    for (int64_t base = ((int64_t)blockIdx.x * (kAnyThreads / 32) + (threadIdx.x >> 5)) * (32 * P); base < pieces; base += step) {
        const int64_t fb = 16 * base - mis > 0 ? 16 * base - mis : 0;            // the step's first byte of the matrix
        const int64_t r0 = quotient(fb, cols), c0 = fb - r0 * cols;
        const uint32_t* const row = packed + r0 * words;
        uint32_t lo[P], hi[P];
        bool whole[P];                                                           // in one row
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const int64_t f = 16 * (base + 32 * k + lane) - mis;                 // the piece's first byte, below 0 in the first
            int64_t c = c0;
            const uint32_t dr = advance(c, f < fb ? 0 : (int)(f - fb), cols);
            whole[k] = f >= 0 && f + 16 <= bytes && c + 16 <= cols;
            const uint32_t* const src = row + dr * words + (c >> 5);
            lo[k] = whole[k] ? __ldg(src) : 0u;
            hi[k] = whole[k] && (c & 31) > 16 ? __ldg(src + 1) : 0u;
        }
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const int64_t f = 16 * (base + 32 * k + lane) - mis;
            int64_t c = c0;
            uint32_t dr = advance(c, f < fb ? 0 : (int)(f - fb), cols);
            uint4* const dst = reinterpret_cast<uint4*>(w + f);
            if (whole[k]) {
                const uint32_t a = convert_order(lo[k], order, NQ_LSB_FIRST), b = convert_order(hi[k], order, NQ_LSB_FIRST);
                __stcs(dst, signs_of16(__funnelshift_r(a, b, (uint32_t)c & 31u)));
            } else if (f < bytes) {
                const int first = f < 0 ? (int)-f : 0, end = bytes - f < 16 ? (int)(bytes - f) : 16;
                uint32_t h = 0;
                for (int e = first; e < end;) {
                    int n = 32 - (int)(c & 31);
                    n = n < end - e ? n : end - e;
                    n = cols - c < n ? (int)(cols - c) : n;
                    const uint32_t word = convert_order(__ldg(row + dr * words + (c >> 5)), order, NQ_LSB_FIRST);
                    h |= ((word >> (c & 31)) & ((1u << n) - 1u)) << e;           // n <= 16
                    e += n; c += n;
                    if (c == cols) { c = 0; ++dr; }
                }
                if (end - first == 16) __stcs(dst, signs_of16(h));
                else
                    for (int e = first; e < end; ++e) w[f + e] = ((h >> e) & 1u) ? (int8_t)-1 : (int8_t)1;
            }
        }
    }
}

// The same two conversions for matrices of whole 32-column words at a 16-byte aligned address, with every global
// access of a warp contiguous: the dense side moves in 512-byte pieces (one 16-byte piece per lane), the packed
// side in 128-byte pieces (one word per lane), and the lanes trade their halves with shuffles.  A warp handles
// 32 consecutive words (1 KB of weights) per step; `n_words` is a multiple of 32 here, the tail goes to the
// kernels above.
__global__ void __launch_bounds__(256) pack_rows_warp_kernel(const uint4* __restrict__ w, uint32_t* __restrict__ out,
                                                             int64_t n_words, int order) {
    enter();
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32; base < n_words; base += warps * 32) {
        // piece p (16 weights) of this step belongs to word base + p/2, half p & 1
        const uint4 a = __ldcs(w + base * 2 + lane), b = __ldcs(w + base * 2 + 32 + lane);
        const uint32_t ha = sign_nibble(a.x) | (sign_nibble(a.y) << 4) | (sign_nibble(a.z) << 8) | (sign_nibble(a.w) << 12);
        const uint32_t hb = sign_nibble(b.x) | (sign_nibble(b.y) << 4) | (sign_nibble(b.z) << 8) | (sign_nibble(b.w) << 12);
        // lane L wants word base + L: its halves are pieces 2L and 2L + 1, i.e. lanes 2(L & 15) and +1 of load a (L < 16) or b
        const int src = 2 * (lane & 15);
        const uint32_t a_lo = __shfl_sync(0xffffffffu, ha, src), a_hi = __shfl_sync(0xffffffffu, ha, src + 1);
        const uint32_t b_lo = __shfl_sync(0xffffffffu, hb, src), b_hi = __shfl_sync(0xffffffffu, hb, src + 1);
        const uint32_t bits = lane < 16 ? (a_lo | (a_hi << 16)) : (b_lo | (b_hi << 16));
        out[base + lane] = convert_order(bits, NQ_LSB_FIRST, order);
    }
}

__global__ void __launch_bounds__(256) unpack_rows_warp_kernel(const uint32_t* __restrict__ packed, uint4* __restrict__ w,
                                                               int64_t n_words, int order) {
    enter();
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32; base < n_words; base += warps * 32) {
        const uint32_t mine = convert_order(__ldcs(packed + base + lane), order, NQ_LSB_FIRST);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            // piece 32k + lane: word base + 16k + lane/2, half lane & 1
            const uint32_t word = __shfl_sync(0xffffffffu, mine, 16 * k + (lane >> 1));
            const uint32_t h = (word >> (16 * (lane & 1))) & 0xFFFFu;
            uint32_t v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = 0x01010101u + spread_nibble(h >> (4 * q)) * 0xFEu;   // +1 = 0x01, -1 = 0xFF
            __stcs(w + base * 2 + 32 * k + lane, make_uint4(v[0], v[1], v[2], v[3]));
        }
    }
}

__global__ void reorder_words_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                     int64_t n, int from, int to) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = convert_order(in[i], from, to);
}
// the same with 16-byte accesses (n4 groups of four words, both pointers 16-byte aligned)
__global__ void reorder_words4_kernel(const uint4* __restrict__ in, uint4* __restrict__ out, int64_t n4, int from, int to) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n4;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint4 v = __ldg(in + i);
        out[i] = make_uint4(convert_order(v.x, from, to), convert_order(v.y, from, to), convert_order(v.z, from, to),
                            convert_order(v.w, from, to));
    }
}

// ---------------------------------------------------------------------------
// marlin layout.  out = 64*to + 16*o16 + 8*o8 + o1, in = 16*tr + 8*r8 + 2*r2 + r1
//   word (tr, 32*to + 4*o1 + r2), bit 15 - 4*o16 - 2*o8 - r8 + 16*r1
// ---------------------------------------------------------------------------
__global__ void pack_marlin_kernel(const int8_t* __restrict__ w, uint32_t* __restrict__ B,
                                   int64_t out_f, int64_t in_f) {
    const int64_t ncol = out_f / 2, total = (in_f / 16) * ncol;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t tr = i / ncol, col = i - tr * ncol;
        const int64_t to = col >> 5;
        const int o1 = (int)(col & 31) >> 2, r2 = (int)(col & 3);
        uint32_t bits = 0;
#pragma unroll
        for (int o16 = 0; o16 < 4; ++o16)
#pragma unroll
            for (int o8 = 0; o8 < 2; ++o8)
#pragma unroll
                for (int r8 = 0; r8 < 2; ++r8) {
                    const int64_t o = 64 * to + 16 * o16 + 8 * o8 + o1;
                    const int64_t k = 16 * tr + 8 * r8 + 2 * r2;
                    const int8_t* p = w + o * in_f + k;
                    const int pos = 15 - 4 * o16 - 2 * o8 - r8;
                    bits |= (uint32_t)(p[0] < 0) << pos;
                    bits |= (uint32_t)(p[1] < 0) << (pos + 16);
                }
        B[i] = bits;
    }
}

// The same through shared memory: a CTA stages 64 output rows x 128 input columns with 16-byte row loads (a row
// segment of 128 bytes is one coalesced request) and every thread assembles one word of the 8 x 32 words of the
// tile from it.  The direct kernel above reads two single bytes per bit pair at a stride of in_f bytes.
constexpr int kMarlinKT = 128;              // input columns per CTA
constexpr int kMarlinPitch = kMarlinKT + 16;
__global__ void __launch_bounds__(256) pack_marlin_staged_kernel(const int8_t* __restrict__ w, uint32_t* __restrict__ B,
                                                                 int64_t out_f, int64_t in_f) {
    __shared__ __align__(16) int8_t tile[64 * kMarlinPitch];
    const int64_t to = blockIdx.x, k0 = (int64_t)blockIdx.y * kMarlinKT;
    const int t = threadIdx.x;
    for (int idx = t; idx < 64 * (kMarlinKT / 16); idx += 256) {
        const int row = idx / (kMarlinKT / 16), seg = idx % (kMarlinKT / 16);
        if (k0 + 16 * seg < in_f)      // in_f is a multiple of 16: a segment is inside the row or beyond it as a whole
            *reinterpret_cast<uint4*>(tile + row * kMarlinPitch + 16 * seg) =
                __ldg(reinterpret_cast<const uint4*>(w + (64 * to + row) * in_f + k0 + 16 * seg));
    }
    __syncthreads();
    const int trl = t >> 5, colw = t & 31;
    if (k0 + 16 * trl >= in_f) return;
    const int o1 = colw >> 2, r2 = colw & 3;
    uint32_t bits = 0;
#pragma unroll
    for (int o16 = 0; o16 < 4; ++o16)
#pragma unroll
        for (int o8 = 0; o8 < 2; ++o8)
#pragma unroll
            for (int r8 = 0; r8 < 2; ++r8) {
                // the two weights of a bit pair are neighbours: one 16-bit load, sign bits 7 and 15 -> pos and pos + 16
                const uint32_t h = *reinterpret_cast<const uint16_t*>(tile + (16 * o16 + 8 * o8 + o1) * kMarlinPitch +
                                                                      16 * trl + 8 * r8 + 2 * r2);
                const int pos = 15 - 4 * o16 - 2 * o8 - r8;
                bits |= (((h >> 7) & 1u) | ((h << 1) & 0x10000u)) << pos;
            }
    B[(k0 / 16 + trl) * (out_f / 2) + 32 * to + colw] = bits;
}

__global__ void marlin_to_rows_kernel(const uint32_t* __restrict__ B, uint32_t* __restrict__ packed,
                                      int64_t out_f, int64_t in_f, int order) {
    const int64_t words = in_f / 32, total = out_f * words, ncol = out_f / 2;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = i / words, wi = i - o * words;
        const int64_t to = o >> 6;
        const int o16 = (int)(o >> 4) & 3, o8 = (int)(o >> 3) & 1, o1 = (int)o & 7;
        uint32_t bits = 0;
#pragma unroll
        for (int t = 0; t < 2; ++t) {  // two k-tiles of 16 per 32-column word
            const int64_t tr = wi * 2 + t;
#pragma unroll
            for (int r2 = 0; r2 < 4; ++r2) {
                const uint32_t src = B[tr * ncol + 32 * to + 4 * o1 + r2];
#pragma unroll
                for (int r8 = 0; r8 < 2; ++r8)
#pragma unroll
                    for (int r1 = 0; r1 < 2; ++r1) {
                        const int pos = 15 - 4 * o16 - 2 * o8 - r8 + 16 * r1;
                        const int k = 16 * t + 8 * r8 + 2 * r2 + r1;
                        bits |= ((src >> pos) & 1u) << k;
                    }
            }
        }
        packed[i] = convert_order(bits, NQ_LSB_FIRST, order);
    }
}

// kind 0: groups of 16, new[4b+2a+c] = old[8a+2b+c]; kind 1: groups of 32, new[8b+2a+c] = old[8a+2b+c]
__global__ void permute_scale16_kernel(const uint16_t* __restrict__ s, uint16_t* __restrict__ out,
                                       int64_t n, int kind, int inverse) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t base;
        int p, a, b, c, src;
        if (kind == 0) {
            base = i & ~15LL; p = (int)(i & 15);
            b = p >> 2; a = (p >> 1) & 1; c = p & 1;   // p = 4b + 2a + c
            src = 8 * a + 2 * b + c;
        } else {
            base = i & ~31LL; p = (int)(i & 31);
            b = p >> 3; a = (p >> 1) & 3; c = p & 1;   // p = 8b + 2a + c
            src = 8 * a + 2 * b + c;
        }
        if (!inverse) out[i] = s[base + src];
        else out[base + src] = s[i];
    }
}

// ---------------------------------------------------------------------------
// tile layout of the GEMV kernel
//
// A tile covers 16 rows x 256 columns and is stored as 32 lanes x uint4 (512 B),
// tiles ordered [row_group][chunk].  Lane l = 4*g + q holds
//   .x: row g,   columns half h=0      .y: row g+8, h=0
//   .z: row g,   h=1                   .w: row g+8, h=1
// and inside a word the weight of column 32*j + 16*h + 4*q + b (of the chunk)
// sits at bit 8*b + j.  `word & (0x01010101 << j)` is then directly the int8
// A-fragment register of an m16n8k32 MMA over columns [32j, 32j+32) with values
// {0, 2^j} (j = 7: {0, -128}).  Rows and columns beyond the matrix are +1 (bit 0).
// ---------------------------------------------------------------------------
// A warp per tile: its 16 pieces of 32 bytes come in with four loads of four pieces each (the neighbouring warp's tile has the
// rest of a line), are turned around in shared memory and leave as one contiguous store.  Tiles are dealt one by one, so
// that a matrix of any number of chunks keeps every warp busy: blocks of eight chunks of a row group, which had idle warps
// at ragged ends and a block barrier, took 6.1 us for 12288 x 2432, this takes 4.7.
__global__ void __launch_bounds__(256) rows_to_tiles_kernel(const uint32_t* __restrict__ packed, uint4* __restrict__ tiles,
                                                            int64_t rows, int64_t words, int64_t chunks, int64_t n_tiles, int order) {
    enter();
    __shared__ uint32_t s[8][16 * 9];
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    uint32_t* const mine = s[threadIdx.x >> 5];
    const int64_t step = (int64_t)gridDim.x * 8;
    for (int64_t tile = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); tile < n_tiles; tile += step) {
        const int64_t rg = quotient(tile, chunks), wi = (tile - rg * chunks) * 8 + (lane & 7), r0 = rg * 16 + (lane >> 3);
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = r0 + 4 * k < rows && wi < words ? __ldg(packed + (r0 + 4 * k) * words + wi) : 0u;
        __syncwarp();       // the previous tile has been read
#pragma unroll
        for (int k = 0; k < 4; ++k)   // padding words are 0 in either order
            mine[(4 * k + (lane >> 3)) * 9 + (lane & 7)] = convert_order(v[k], order, NQ_LSB_FIRST);
        __syncwarp();
        uint32_t o[4] = {0, 0, 0, 0};
#pragma unroll
        for (int half_row = 0; half_row < 2; ++half_row)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t src = mine[(g + 8 * half_row) * 9 + j];
                o[half_row] |= spread_nibble(src >> (4 * q)) << j;           // h = 0
                o[2 + half_row] |= spread_nibble(src >> (16 + 4 * q)) << j;  // h = 1
            }
        __stcs(tiles + tile * 32 + lane, make_uint4(o[0], o[1], o[2], o[3]));
    }
}

__global__ void tiles_to_rows_kernel(const uint4* __restrict__ tiles, uint32_t* __restrict__ packed,
                                     int64_t rows, int64_t words, int64_t chunks, int order) {
    const int64_t total = rows * words;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / words, wi = i - r * words;
        const int64_t rg = r >> 4, c = wi >> 3;
        const int g = (int)(r & 7), half_row = (int)(r >> 3) & 1, j = (int)(wi & 7);
        uint32_t bits = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint4 t = tiles[(rg * chunks + c) * 32 + 4 * g + q];
            const uint32_t lo = half_row ? t.y : t.x, hi = half_row ? t.w : t.z;
            const uint32_t nlo = (((lo >> j) & 0x01010101u) * 0x01020408u) >> 24;
            const uint32_t nhi = (((hi >> j) & 0x01010101u) * 0x01020408u) >> 24;
            bits |= (nlo & 0xFu) << (4 * q);
            bits |= (nhi & 0xFu) << (16 + 4 * q);
        }
        packed[i] = convert_order(bits, NQ_LSB_FIRST, order);
    }
}

// gcd(n, 32) for n > 0: the largest power of two up to 32 that divides n
static int64_t gcd32(int64_t n) {
    int64_t g = 1;
    while (g < 32 && n % (2 * g) == 0) g *= 2;
    return g;
}

static int check_order(int o) { return (o == NQ_LSB_FIRST || o == NQ_HALF2) ? NQ_OK : NQ_ERR_DTYPE; }

}  // namespace nq

using namespace nq;

extern "C" {

int nq_pack_rows(const int8_t* w, int32_t* packed, int64_t rows, int64_t cols, int bit_order,
                 nq_stream_t stream) {
    if (rows < 0 || cols < 0) return NQ_ERR_SHAPE;
    if (check_order(bit_order) != NQ_OK) return NQ_ERR_DTYPE;
    if (rows == 0 || cols == 0) return NQ_OK;
    if (!w || !packed) return NQ_ERR_NULL;
    const int64_t words = (cols + 31) / 32;
    uint32_t* const out = reinterpret_cast<uint32_t*>(packed);
    // whole words at an aligned address: the rows form one run of words; the leading rows whose words are a multiple
    // of 32 go to the kernel without index arithmetic, the remaining rows to the general one
    int64_t done = 0;
    if (cols % 32 == 0 && aligned16(w)) {
        const int64_t step = 32 / gcd32(words), head_rows = rows / step * step, head = head_rows * words;
        if (head > 0) {
            const int st = launch(pack_rows_warp_kernel, grid_for(head, kPackThreads), kPackThreads, stream,
                                  reinterpret_cast<const uint4*>(w), out, head, bit_order);
            if (st != NQ_OK) return st;
            done = head_rows;
        }
    }
    if (done == rows) return NQ_OK;
    return launch(pack_rows_kernel, grid_for(((rows - done) * words + 1) / 2, kAnyThreads), kAnyThreads, stream, w + done * cols,
                  out + done * words, rows - done, cols, words, bit_order);
}

int nq_unpack_rows(const int32_t* packed, int8_t* w, int64_t rows, int64_t cols, int bit_order,
                   nq_stream_t stream) {
    if (rows < 0 || cols < 0) return NQ_ERR_SHAPE;
    if (check_order(bit_order) != NQ_OK) return NQ_ERR_DTYPE;
    if (rows == 0 || cols == 0) return NQ_OK;
    if (!w || !packed) return NQ_ERR_NULL;
    const int64_t words = (cols + 31) / 32;
    const uint32_t* const in = reinterpret_cast<const uint32_t*>(packed);
    int64_t done = 0;
    if (cols % 32 == 0 && aligned16(w)) {   // see nq_pack_rows
        const int64_t step = 32 / gcd32(words), head_rows = rows / step * step, head = head_rows * words;
        if (head > 0) {
            const int st = launch(unpack_rows_warp_kernel, grid_for(head, kPackThreads), kPackThreads, stream, in,
                                  reinterpret_cast<uint4*>(w), head, bit_order);
            if (st != NQ_OK) return st;
            done = head_rows;
        }
    }
    if (done == rows) return NQ_OK;
    // Four pieces per lane share the row arithmetic and are in flight together (12291 x 2435: 13.8 us with two, 12.5 with
    // four), where that leaves every SM a few blocks; else one (1000 x 777: 3.3 us with four).
    const int64_t pieces = ((rows - done) * cols + 15) / 16 + 1;
    const bool many = pieces >= (int64_t)sm_count() * 8 * kAnyThreads * 4;
    return launch(many ? unpack_rows_kernel<4> : unpack_rows_kernel<1>, grid_for(many ? (pieces + 3) / 4 : pieces, kAnyThreads),
                  kAnyThreads, stream, in + done * words, w + done * cols, rows - done, cols, words, bit_order);
}

int nq_reorder_words(const int32_t* in, int32_t* out, int64_t n_words, int order_in, int order_out,
                     nq_stream_t stream) {
    if (n_words < 0) return NQ_ERR_SHAPE;
    if (check_order(order_in) != NQ_OK || check_order(order_out) != NQ_OK) return NQ_ERR_DTYPE;
    if (n_words == 0) return NQ_OK;
    if (!in || !out) return NQ_ERR_NULL;
    if (n_words % 4 == 0 && aligned16(in) && aligned16(out))
        reorder_words4_kernel<<<grid_for(n_words / 4, kPackThreads), kPackThreads, 0, as_stream(stream)>>>(
            reinterpret_cast<const uint4*>(in), reinterpret_cast<uint4*>(out), n_words / 4, order_in, order_out);
    else
        reorder_words_kernel<<<grid_for(n_words, kPackThreads), kPackThreads, 0, as_stream(stream)>>>(
            reinterpret_cast<const uint32_t*>(in), reinterpret_cast<uint32_t*>(out), n_words, order_in, order_out);
    NQ_LAUNCH_CHECK();
    return NQ_OK;
}

int nq_pack_marlin(const int8_t* w, int32_t* B, int64_t out_f, int64_t in_f, nq_stream_t stream) {
    if (out_f < 0 || in_f < 0 || out_f % 64 || in_f % 16) return NQ_ERR_SHAPE;
    if (out_f == 0 || in_f == 0) return NQ_OK;
    if (!w || !B) return NQ_ERR_NULL;
    const int64_t kblocks = (in_f + kMarlinKT - 1) / kMarlinKT;
    if (aligned16(w) && out_f / 64 <= 0x7FFFFFFF && kblocks <= 65535)
        pack_marlin_staged_kernel<<<dim3((unsigned)(out_f / 64), (unsigned)kblocks), 256, 0, as_stream(stream)>>>(
            w, reinterpret_cast<uint32_t*>(B), out_f, in_f);
    else
        pack_marlin_kernel<<<grid_for((in_f / 16) * (out_f / 2), kPackThreads), kPackThreads, 0, as_stream(stream)>>>(
            w, reinterpret_cast<uint32_t*>(B), out_f, in_f);
    NQ_LAUNCH_CHECK();
    return NQ_OK;
}

int nq_marlin_to_rows(const int32_t* B, int32_t* packed, int64_t out_f, int64_t in_f, int bit_order,
                      nq_stream_t stream) {
    if (out_f < 0 || in_f < 0 || out_f % 64 || in_f % 32) return NQ_ERR_SHAPE;
    if (check_order(bit_order) != NQ_OK) return NQ_ERR_DTYPE;
    if (out_f == 0 || in_f == 0) return NQ_OK;
    if (!B || !packed) return NQ_ERR_NULL;
    marlin_to_rows_kernel<<<grid_for(out_f * (in_f / 32), kPackThreads), kPackThreads, 0, as_stream(stream)>>>(
        reinterpret_cast<const uint32_t*>(B), reinterpret_cast<uint32_t*>(packed), out_f, in_f, bit_order);
    NQ_LAUNCH_CHECK();
    return NQ_OK;
}

int nq_permute_scale16(const void* s, void* out, int64_t n, int kind, int inverse, nq_stream_t stream) {
    if (kind != 0 && kind != 1) return NQ_ERR_DTYPE;
    if (n < 0 || n % (kind == 0 ? 16 : 32)) return NQ_ERR_SHAPE;
    if (n == 0) return NQ_OK;
    if (!s || !out) return NQ_ERR_NULL;
    if (s == out) return NQ_ERR_UNSUPPORTED;  // not an in-place permutation
    permute_scale16_kernel<<<grid_for(n, kPackThreads), kPackThreads, 0, as_stream(stream)>>>(
        static_cast<const uint16_t*>(s), static_cast<uint16_t*>(out), n, kind, inverse);
    NQ_LAUNCH_CHECK();
    return NQ_OK;
}

size_t nq_tiles_bytes(int64_t rows, int64_t cols) {
    if (rows <= 0 || cols <= 0) return 0;
    return (size_t)((rows + 15) / 16) * (size_t)((cols + 255) / 256) * 512;
}

int nq_rows_to_tiles(const int32_t* packed, void* tiles, int64_t rows, int64_t cols, int bit_order,
                     nq_stream_t stream) {
    if (rows <= 0 || cols <= 0) return NQ_ERR_SHAPE;
    if (check_order(bit_order) != NQ_OK) return NQ_ERR_DTYPE;
    if (!packed || !tiles) return NQ_ERR_NULL;
    if (!aligned16(tiles)) return NQ_ERR_ALIGN;
    const int64_t words = (cols + 31) / 32, chunks = (cols + 255) / 256, n_tiles = (rows + 15) / 16 * chunks;
    return launch(rows_to_tiles_kernel, grid_for(n_tiles * 32, 256), 256, stream, reinterpret_cast<const uint32_t*>(packed),
                  static_cast<uint4*>(tiles), rows, words, chunks, n_tiles, bit_order);
}

int nq_tiles_to_rows(const void* tiles, int32_t* packed, int64_t rows, int64_t cols, int bit_order,
                     nq_stream_t stream) {
    if (rows <= 0 || cols <= 0) return NQ_ERR_SHAPE;
    if (check_order(bit_order) != NQ_OK) return NQ_ERR_DTYPE;
    if (!packed || !tiles) return NQ_ERR_NULL;
    if (!aligned16(tiles)) return NQ_ERR_ALIGN;
    const int64_t words = (cols + 31) / 32, chunks = (cols + 255) / 256;
    tiles_to_rows_kernel<<<grid_for(rows * words, kPackThreads), kPackThreads, 0, as_stream(stream)>>>(
        static_cast<const uint4*>(tiles), reinterpret_cast<uint32_t*>(packed), rows, words, chunks, bit_order);
    NQ_LAUNCH_CHECK();
    return NQ_OK;
}

}  // extern "C"
