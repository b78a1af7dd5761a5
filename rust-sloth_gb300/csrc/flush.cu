// flush.cu -- the bytes Context::flush prints, formatted on the GPU from the frame cells.
//
// src/context.rs:50-92.  For a frame of cells (char | r<<8 | g<<16 | b<<24):
//   - terminal contexts (image false) first queue crossterm's MoveTo(0,0): ESC "[1;1H";
//   - color false: every char, then println's "\n";
//   - color true, webify false: per cell crossterm 0.18's PrintStyledContent of the char
//     with foreground Rgb(r,g,b) on background Rgb(25,25,25):
//       ESC "[48;2;25;25;25m" ESC "[38;2;<r>;<g>;<b>m" <char> ESC "[0m"
//     (crossterm 0.18.0 is the version Cargo.lock pins; its source is not in the reference
//     tree, so this sequence restates its published StyledContent output: background,
//     foreground, content, ResetColor);
//   - color true, webify true: per cell "<span style=\"color:rgb(<r>,<g>,<b>)\"><char>".
// Numbers are decimal without padding.
//
// Three launches: per-chunk byte counts, one block scanning the chunk counts, and the
// formatter, which builds each chunk's text in shared memory and writes it out in one
// contiguous run.  A call that only asks for the size stops after the scan.
#include <cstdint>

#include "flush_kernels.h"
#include "sloth_internal.cuh"

namespace sloth {

namespace {

constexpr int kFlushThreads = 256;
constexpr int kFlushCellsPerThread = 4;
constexpr uint32_t kFlushChunk = kFlushThreads * kFlushCellsPerThread;   // cells per block
constexpr uint32_t kMaxCellBytes = 40;                                      // ANSI: 31 + 9 digits

__device__ __forceinline__ uint32_t ndigits(uint32_t v) { return v >= 100 ? 3u : (v >= 10 ? 2u : 1u); }

__device__ __forceinline__ uint32_t cell_bytes(uint32_t cell, int format)
{
    if (format == kFlushPlain) return 1;
    const uint32_t d = ndigits((cell >> 8) & 255u) + ndigits((cell >> 16) & 255u) + ndigits(cell >> 24);
    return format == kFlushAnsi ? 31u + d : 29u + d;
}

// Appends bytes to a run of shared text, a word at a time: the bytes collect in a 64-bit
// register and leave as whole words, so a cell costs about ten stores instead of forty.
// The first and last words of a thread's run are shared with its neighbours' and are
// written by bytes.
struct Emit {
    char *text;
    uint32_t pos;     // byte position of the collected bytes' word (a multiple of 4)
    uint32_t fill;    // bytes in the register, those before the run's start included
    uint32_t skip;    // bytes of the first word that belong to the run before
    uint64_t acc;

    __device__ __forceinline__ Emit(char *t, uint32_t off) : text(t), pos(off & ~3u), fill(off & 3u), skip(off & 3u), acc(0) {}
    // n bytes (1..4) from the low end of w; the bytes above them are zero
    __device__ __forceinline__ void put(uint32_t w, uint32_t n)
    {
        acc |= (uint64_t)w << (8 * fill);
        fill += n;
        if (fill >= 4) {
            if (skip) {
                for (uint32_t k = skip; k < 4; ++k) text[pos + k] = (char)(acc >> (8 * k));
                skip = 0;
            } else {
                *reinterpret_cast<uint32_t *>(text + pos) = (uint32_t)acc;
            }
            acc >>= 32;
            pos += 4;
            fill -= 4;
        }
    }
    __device__ __forceinline__ void end()
    {
        for (uint32_t k = skip; k < fill; ++k) text[pos + k] = (char)(acc >> (8 * k));
    }
    // a decimal number (0..255) and the character after it
    __device__ __forceinline__ void number(uint32_t v, uint32_t after)
    {
        const uint32_t h = v / 100, t = v / 10 - 10 * h, u = v - 10 * (v / 10);
        const uint32_t n = ndigits(v);
        const uint32_t d = n == 3 ? (h | t << 8 | u << 16) + 0x303030u : n == 2 ? (t | u << 8) + 0x3030u : u + 0x30u;
        put(d | after << (8 * n), n + 1);
    }
};

__host__ __device__ constexpr uint32_t word4(const char *s)
{
    return (uint32_t)(uint8_t)s[0] | (uint32_t)(uint8_t)s[1] << 8 | (uint32_t)(uint8_t)s[2] << 16 |
           (uint32_t)(uint8_t)s[3] << 24;
}
__host__ __device__ constexpr uint32_t word3(const char *s)
{
    return (uint32_t)(uint8_t)s[0] | (uint32_t)(uint8_t)s[1] << 8 | (uint32_t)(uint8_t)s[2] << 16;
}

__device__ __forceinline__ void put_cell(Emit &o, uint32_t cell, int format)
{
    const uint32_t ch = cell & 255u;
    if (format == kFlushPlain) {
        o.put(ch, 1);
        return;
    }
    const uint32_t r = (cell >> 8) & 255u, g = (cell >> 16) & 255u, b = cell >> 24;
    if (format == kFlushAnsi) {
        constexpr uint32_t w0 = word4("\x1b[48"), w1 = word4(";2;2"), w2 = word4("5;25"), w3 = word4(";25m"),
                           w4 = word4("\x1b[38"), w5 = word3(";2;"), w6 = word3("\x1b[0");
        o.put(w0, 4); o.put(w1, 4); o.put(w2, 4); o.put(w3, 4); o.put(w4, 4); o.put(w5, 3);
        o.number(r, ';');
        o.number(g, ';');
        o.number(b, 'm');
        o.put(ch | w6 << 8, 4);
        o.put('m', 1);
    } else {
        constexpr uint32_t w0 = word4("<spa"), w1 = word4("n st"), w2 = word4("yle="), w3 = word4("\"col"),
                           w4 = word4("or:r"), w5 = word3("gb(");
        o.put(w0, 4); o.put(w1, 4); o.put(w2, 4); o.put(w3, 4); o.put(w4, 4); o.put(w5, 3);
        o.number(r, ',');
        o.number(g, ',');
        o.number(b, ')');
        o.put((uint32_t)'"' | (uint32_t)'>' << 8 | ch << 16, 3);
    }
}

// Block-wide exclusive scan of one value per thread; returns the prefix, *total the sum.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *ws, uint32_t *total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += o;
    }
    if (lane == 31) ws[wid] = x;
    block_sync();
    if (wid == 0) {
        uint32_t s = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= d) s += o;
        }
        ws[lane] = s;
    }
    block_sync();
    *total = ws[(blockDim.x >> 5) - 1];
    const uint32_t pre = x - v + (wid > 0 ? ws[wid - 1] : 0u);
    block_sync();   // ws may be reused by the caller
    return pre;
}

__global__ void __launch_bounds__(kFlushThreads)
flush_count_kernel(const uint32_t *__restrict__ cells, uint64_t ncells, int format, uint64_t *__restrict__ chunk_bytes)
{
    __shared__ uint32_t ws[32];
    const uint64_t c0 = (uint64_t)blockIdx.x * kFlushChunk + (uint64_t)threadIdx.x * kFlushCellsPerThread;
    uint32_t n = 0;
#pragma unroll
    for (int k = 0; k < kFlushCellsPerThread; ++k)
        if (c0 + k < ncells) n += cell_bytes(cells[c0 + k], format);
    uint32_t total;
    block_exclusive_scan(n, ws, &total);
    if (threadIdx.x == 0) chunk_bytes[blockIdx.x] = total;
}

// One block: exclusive scan of the chunk byte counts in place (64-bit), then the total
// output size (prefix + chunks + trailing newline) into *size.
__global__ void __launch_bounds__(1024)
flush_scan_kernel(uint64_t *__restrict__ chunk_bytes, uint32_t nchunks, uint32_t prefix, uint32_t suffix,
                  uint64_t *__restrict__ size)
{
    __shared__ unsigned long long ws[32];
    __shared__ unsigned long long carry;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = prefix;
    block_sync();
    for (uint32_t base = 0; base < nchunks; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const unsigned long long v = i < nchunks ? chunk_bytes[i] : 0ull;
        unsigned long long x = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long o = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += o;
        }
        if (lane == 31) ws[wid] = x;
        block_sync();
        if (wid == 0) {
            unsigned long long s = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0ull;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long o = __shfl_up_sync(0xffffffffu, s, d);
                if (lane >= d) s += o;
            }
            ws[lane] = s;
        }
        block_sync();
        const unsigned long long pre = carry + x - v + (wid > 0 ? ws[wid - 1] : 0ull);
        if (i < nchunks) chunk_bytes[i] = pre;
        block_sync();
        if (threadIdx.x == blockDim.x - 1) carry = pre + v;
        block_sync();
    }
    if (threadIdx.x == 0) *size = carry + suffix;
}

// Each block formats its chunk into shared memory, then copies it out: the text starts at
// the place in shared memory that its destination has in a 16-byte line, so that all but
// the ends go out in 16-byte stores.  The ends of the whole text (a terminal's MoveTo, the
// line feed of the plain form) are the first and last blocks'.  230k cells of HTML took
// 39 us with byte stores, in shared memory and out of it, and 13 us as here.
__global__ void __launch_bounds__(kFlushThreads)
flush_write_kernel(const uint32_t *__restrict__ cells, uint64_t ncells, int format,
                   const uint64_t *__restrict__ chunk_off, char *__restrict__ out, int image, int suffix)
{
    __shared__ uint32_t ws[32];
    __shared__ __align__(16) char text[kFlushChunk * kMaxCellBytes + 16];
    const uint64_t c0 = (uint64_t)blockIdx.x * kFlushChunk + (uint64_t)threadIdx.x * kFlushCellsPerThread;
    uint32_t cv[kFlushCellsPerThread];
    uint32_t n = 0;
#pragma unroll
    for (int k = 0; k < kFlushCellsPerThread; ++k) {
        cv[k] = c0 + k < ncells ? cells[c0 + k] : 0u;
        if (c0 + k < ncells) n += cell_bytes(cv[k], format);
    }
    uint32_t total;
    const uint32_t off = block_exclusive_scan(n, ws, &total);
    char *dst = out + chunk_off[blockIdx.x];
    const uint32_t lead = (uint32_t)reinterpret_cast<uintptr_t>(dst) & 15u;
    Emit o(text, lead + off);
#pragma unroll
    for (int k = 0; k < kFlushCellsPerThread; ++k)
        if (c0 + k < ncells) put_cell(o, cv[k], format);
    o.end();
    block_sync();
    // bytes [lead, lead + total) of text: line i of 16 bytes starts at dst - lead + 16*i
    char *line0 = dst - lead;
    const uint32_t last = lead + total;
    for (uint32_t i = threadIdx.x; 16 * i < last; i += blockDim.x) {
        const uint32_t b0 = 16 * i;
        if (b0 >= lead && b0 + 16 <= last) {
            reinterpret_cast<uint4 *>(line0)[i] = reinterpret_cast<const uint4 *>(text)[i];
        } else {
            for (uint32_t k = max(b0, lead); k < min(b0 + 16, last); ++k) line0[k] = text[k];
        }
    }
    if (threadIdx.x == 0) {
        if (blockIdx.x == 0 && !image) {
            const char move[6] = {'\x1b', '[', '1', ';', '1', 'H'};
            for (int k = 0; k < 6; ++k) out[k] = move[k];
        }
        if (blockIdx.x == gridDim.x - 1 && suffix) dst[total] = '\n';
    }
}

}  // namespace

uint32_t flush_chunks(uint64_t ncells)
{
    return (uint32_t)((ncells + kFlushChunk - 1) / kFlushChunk);
}

uint64_t flush_max_bytes(uint64_t ncells)
{
    return 6 + ncells * kMaxCellBytes + 1;
}

cudaError_t launch_flush(const uint32_t *cells, uint64_t ncells, int image, int format, uint64_t *chunk_bytes,
                         uint64_t *size, char *out, cudaStream_t s)
{
    const uint32_t nch = flush_chunks(ncells);
    const uint32_t prefix = image ? 0u : 6u;
    const uint32_t suffix = format == kFlushPlain ? 1u : 0u;
    if (nch) flush_count_kernel<<<nch, kFlushThreads, 0, s>>>(cells, ncells, format, chunk_bytes);
    flush_scan_kernel<<<1, 1024, 0, s>>>(chunk_bytes, nch, prefix, suffix, size);
    if (nch && out)
        flush_write_kernel<<<nch, kFlushThreads, 0, s>>>(cells, ncells, format, chunk_bytes, out, image, (int)suffix);
    return cudaGetLastError();
}

cudaError_t flush_run(FlushScratch &f, const uint32_t *cells, uint64_t ncells, int image, int format, bool text,
                      cudaStream_t s, uint64_t *bytes)
{
    cudaError_t e;
    const size_t nch = flush_chunks(ncells);
    const size_t need = flush_max_bytes(ncells);
    if (!f.size_d) {
        if ((e = cudaMalloc(&f.size_d, sizeof(uint64_t))) != cudaSuccess) return e;
        if ((e = cudaMallocHost(&f.size_h, sizeof(uint64_t))) != cudaSuccess) return e;
    }
    if (nch > f.chunks_cap || !f.chunks) {
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
        if (f.chunks) cudaFree(f.chunks);
        f.chunks = nullptr;
        if ((e = cudaMalloc(&f.chunks, (nch ? nch : 1) * sizeof(uint64_t))) != cudaSuccess) return e;
        f.chunks_cap = nch;
    }
    if (need > f.out_cap || !f.out) {
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
        if (f.out) cudaFree(f.out);
        f.out = nullptr;
        if ((e = cudaMalloc(&f.out, need)) != cudaSuccess) return e;
        f.out_cap = need;
    }
    if ((e = launch_flush(cells, ncells, image, format, f.chunks, f.size_d, text ? f.out : nullptr, s)) != cudaSuccess)
        return e;
    if ((e = cudaMemcpyAsync(f.size_h, f.size_d, sizeof(uint64_t), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
        return e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    *bytes = *f.size_h;
    return cudaSuccess;
}

void flush_release(FlushScratch &f)
{
    if (f.chunks) cudaFree(f.chunks);
    if (f.out) cudaFree(f.out);
    if (f.size_d) cudaFree(f.size_d);
    if (f.size_h) cudaFreeHost(f.size_h);
    f = FlushScratch{};
}

}  // namespace sloth
