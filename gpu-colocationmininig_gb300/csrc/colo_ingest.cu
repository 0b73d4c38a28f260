// colo_ingest.cu -- the point CSV parsed on the device.
//
// populateData (Codes/colocationFinder.cpp:139-254) reads the file serially.
// Here the text after the count line is copied to the device once; one pass
// finds the line ends, and one thread per line parses "fid,x,y" with the
// host reader's rules (std::stoi / std::stof prefix parsing, boost's
// tokenizer).  The parsed coordinates stay on the device as the dataset's
// resident copy.
//
// Exactness: a coordinate is converted on the device only when the decimal
// has at most 19 significant digits and the value is m * 10^e with
// m < 2^53 and |e| <= 22.  With -11 <= e <= 0, as coordinates are written, the
// correctly rounded float comes from one integer quotient and its remainder
// (FP64 divisions are slow here).  Else m and 10^|e| are exact doubles and one IEEE
// multiply or divide gives the correctly rounded double of the decimal
// (Clinger's fast path, "How to read floating point numbers accurately",
// PLDI 1990).  Rounding that double to float is the correctly rounded float
// unless the double lies exactly on a float rounding midpoint, which is
// detected.  Every other line -- a midpoint, more digits, a larger exponent,
// a float outside the normal range, "inf"/"nan"/hex/'+', quotes or escapes --
// is flagged and parsed on the host by the same reader the CPU path uses, so
// results are bit-identical to it.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include <fcntl.h>
#include <sys/mman.h>
#include <sys/stat.h>
#include <unistd.h>

#include "colo_batch.h"
#include "colo_device.cuh"
#include "colo_host.h"

namespace colo {

// Host reader pieces (colo_io.cpp).
bool csv_parse_line(const char* b, const char* e, int32_t* id, float* x, float* y, bool* minus_one,
                    std::string* token);
bool csv_parse_count(const char* b, const char* e, long* n);
bool csv_parse_bounds(const char* b, const char* e, float bounds[4]);

namespace {

enum : uint8_t { L_OK = 0, L_EMPTY = 1, L_HOST = 2, L_BAD = 3, L_MINUS1 = 4 };

constexpr int kNlThreads = 256, kNlSteps = 4;
constexpr uint32_t kNlBytes = 16 * kNlSteps, kNlTile = kNlThreads * kNlBytes;   // a thread's bytes, a block's
constexpr uint32_t kMinLine = 6;   // "0,0,0" and its newline: the shortest point line

// One bit per byte of a 32-bit word that equals '\n' (0x0A), lowest byte first.
__device__ __forceinline__ uint32_t nl_bits(uint32_t w) {
    const uint32_t x = w ^ 0x0A0A0A0Au;
    const uint32_t t = ~(((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) & 0x80808080u;   // high bit of every matching byte
    return (t >> 7) * 0x10204080u >> 28;   // bits 0, 8, 16, 24 to 28 .. 31
}

// Positions of the line ends in one pass: a block marks the newlines of a 16 KB tile
// (a bit a byte, from coalesced 16-byte loads), counts them, takes its place from a
// decoupled look-back and writes as many as nl holds (cap; the total is the last
// tile's status word).  buf is 16-byte aligned and readable up to a multiple of 16.
// Bound by the look-back and the launch at this size: a count, a scan and a
// second read byte by byte took 90 us for 24 MB (1M lines), this 25.
__global__ void __launch_bounds__(kNlThreads) k_line_ends(const uint8_t* __restrict__ buf, uint64_t n,
                                                          unsigned long long* __restrict__ status,
                                                          uint32_t* __restrict__ ticket, uint64_t* __restrict__ nl,
                                                          uint64_t cap) {
    __shared__ uint32_t s_tile;
    __shared__ unsigned long long s_prefix;
    __shared__ __align__(8) uint16_t s_bits[kNlThreads * kNlSteps];
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t t0 = (uint64_t)tile * kNlTile;
#pragma unroll
    for (int i = 0; i < kNlSteps; ++i) {
        const uint32_t at = (uint32_t)i * kNlThreads + threadIdx.x;
        const uint64_t b = t0 + (uint64_t)at * 16;
        uint32_t m = 0;
        if (b < n) {
            const uint4 v = *reinterpret_cast<const uint4*>(buf + b);
            m = nl_bits(v.x) | nl_bits(v.y) << 4 | nl_bits(v.z) << 8 | nl_bits(v.w) << 12;
            if (n - b < 16) m &= (1u << (uint32_t)(n - b)) - 1u;
        }
        s_bits[at] = (uint16_t)m;
    }
    __syncthreads();
    uint64_t mine = reinterpret_cast<const uint64_t*>(s_bits)[threadIdx.x];
    uint32_t tot;
    const uint32_t ex = block_excl_scan<uint32_t>((uint32_t)__popcll(mine), &tot);
    if (threadIdx.x < 32) {
        unsigned long long prefix;
        if (!warp_lookback(status, tile, tot, prefix)) {   // the text before this tile, counted here
            unsigned long long add = 0;
            for (uint64_t b = threadIdx.x; b < t0; b += 32) add += buf[b] == '\n';
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
            prefix = add;
            lookback_publish(status, tile, prefix + tot);
        }
        if (threadIdx.x == 0) s_prefix = prefix;
    }
    __syncthreads();
    uint64_t o = s_prefix + ex;
    const uint64_t b = t0 + (uint64_t)threadIdx.x * kNlBytes;
    for (; mine && o < cap; mine &= mine - 1) nl[o++] = b + (uint64_t)(__ffsll((long long)mine) - 1);
}

__device__ __forceinline__ bool is_space(uint8_t c) {
    return c == ' ' || c == '\t' || c == '\n' || c == '\v' || c == '\f' || c == '\r';
}

// std::stoi on [b, e): 0 ok, 1 malformed.
__device__ int parse_int_dev(const uint8_t* b, const uint8_t* e, int32_t* v) {
    const uint8_t* p = b;
    while (p < e && is_space(*p)) ++p;
    bool neg = false;
    if (p < e && (*p == '+' || *p == '-')) neg = *p++ == '-';
    const uint8_t* d = p;
    int64_t r = 0;
    for (; p < e && *p >= '0' && *p <= '9'; ++p)
        if (r <= (int64_t)INT32_MAX + 1) r = r * 10 + (*p - '0');
    if (p == d) return 1;
    if (neg) r = -r;
    if (r < INT32_MIN || r > INT32_MAX) return 1;
    *v = (int32_t)r;
    return 0;
}

// 10^k, its reciprocal floor(2^(63 + L) / 10^k) with 2^(L-1) < 10^k <= 2^L, and L - 1.
constexpr int kIntDigits = 11;
struct Tenth {
    uint64_t d, inv;
    int shift;
};
constexpr Tenth tenth(int k) {
    uint64_t d = 1;
    for (int i = 0; i < k; ++i) d *= 10;
    int L = 0;
    while ((1ull << L) < d) ++L;
    uint64_t q = 0, r = 1;   // long division of 2^(63 + L), a bit at a time
    for (int i = 0; i < 63 + L; ++i) {
        r <<= 1;
        q <<= 1;
        if (r >= d) {
            r -= d;
            q |= 1;
        }
    }
    return {d, q, L - 1};
}
__constant__ Tenth c_tenth[kIntDigits + 1] = {{1, 0, 0}, tenth(1), tenth(2), tenth(3), tenth(4), tenth(5),
                                              tenth(6),  tenth(7), tenth(8), tenth(9), tenth(10), tenth(11)};
__constant__ double c_p10[23] = {1e0,  1e1,  1e2,  1e3,  1e4,  1e5,  1e6,  1e7,  1e8,  1e9,  1e10, 1e11,
                                 1e12, 1e13, 1e14, 1e15, 1e16, 1e17, 1e18, 1e19, 1e20, 1e21, 1e22};

// The float nearest to m / 10^k (ties to even), m in 1 .. 2^53 - 1, 1 <= k <= kIntDigits, in integers.
// m is shifted to 64 bits, so the quotient has at least 27; the product with the reciprocal,
// which is below 2^(63 + L) / 10^k by less than one, gives it or one less.
__device__ __forceinline__ float decimal_to_float(uint64_t m, int k) {
    const Tenth t = c_tenth[k];
    const int z = __clzll((long long)m);
    const uint64_t num = m << z;
    uint64_t q = __umul64hi(num, t.inv) >> t.shift;
    uint64_t r = num - q * t.d;
    if (r >= t.d) {
        r -= t.d;
        ++q;
    }
    const int drop = 40 - __clzll((long long)q);   // bits of q below the 24 kept
    const uint64_t half = 1ull << (drop - 1), low = q & (2 * half - 1);
    uint32_t mant = (uint32_t)(q >> drop);
    if (low > half || (low == half && (r || (mant & 1u)))) ++mant;
    return ldexpf((float)mant, drop - z);   // exact: 24 bits (2^24 on a carry) in the normal range
}

// std::stof on [b, e) as the host reader does it: 0 converted exactly here,
// 1 left to the host, 2 malformed (no number at the start).
__device__ int parse_float_dev(const uint8_t* b, const uint8_t* e, float* v) {
    const uint8_t* p = b;
    while (p < e && is_space(*p)) ++p;
    for (const uint8_t* q = p; q < e; ++q)
        if (*q == 'x' || *q == 'X') return 1;   // hexadecimal forms: the host
    if (p < e && (*p == '+' || *p == 'i' || *p == 'I' || *p == 'n' || *p == 'N')) return 1;
    bool neg = false;
    if (p < e && *p == '-') {
        neg = true;
        ++p;
        if (p < e && (*p == 'i' || *p == 'I' || *p == 'n' || *p == 'N')) return 1;
    }
    uint64_t m = 0;
    int sig = 0, frac = 0, dropped = 0;
    bool any = false;
    for (; p < e && *p >= '0' && *p <= '9'; ++p) {
        any = true;
        if (m == 0 && *p == '0') continue;
        if (sig < 19) {
            m = m * 10 + (*p - '0');
            ++sig;
        } else {
            ++dropped;
        }
    }
    if (p < e && *p == '.') {
        ++p;
        for (; p < e && *p >= '0' && *p <= '9'; ++p) {
            any = true;
            if (m == 0 && *p == '0') {
                ++frac;
                continue;
            }
            if (sig < 19) {
                m = m * 10 + (*p - '0');
                ++sig;
                ++frac;
            } else {
                ++dropped;   // digits past 19 after the point: the value is not m * 10^e exactly
            }
        }
    }
    if (!any) return 2;
    if (dropped) return 1;
    int ex = 0;
    if (p < e && (*p == 'e' || *p == 'E')) {
        const uint8_t* q = p + 1;
        bool eneg = false;
        if (q < e && (*q == '+' || *q == '-')) eneg = *q++ == '-';
        if (q < e && *q >= '0' && *q <= '9') {   // otherwise the 'e' is not part of the number
            int x = 0;
            for (; q < e && *q >= '0' && *q <= '9'; ++q)
                if (x < 100000) x = x * 10 + (*q - '0');
            ex = eneg ? -x : x;
        }
    }
    if (m == 0) {
        *v = neg ? -0.0f : 0.0f;
        return 0;
    }
    const int e10 = ex - frac;
    if (m >= (1ull << 53) || e10 < -22 || e10 > 22) return 1;
    if (e10 <= 0 && e10 >= -kIntDigits) {
        const float f = e10 == 0 ? __ull2float_rn(m) : decimal_to_float(m, -e10);
        *v = neg ? -f : f;
        return 0;
    }
    const double dm = (double)m;   // exact: m < 2^53
    const double d = e10 >= 0 ? __dmul_rn(dm, c_p10[e10]) : __ddiv_rn(dm, c_p10[-e10]);
    // float normal range only (no subnormal or overflow handling here)
    if (!(d >= 1.1754943508222875e-38) || d > 3.4028234663852886e38) return 1;
    // a float rounding midpoint: the 29 low mantissa bits are exactly 1000...0
    const unsigned long long bits = (unsigned long long)__double_as_longlong(d);
    if ((bits & ((1ull << 29) - 1)) == (1ull << 28)) return 1;
    const float f = __double2float_rn(d);
    *v = neg ? -f : f;
    return 0;
}

__device__ __forceinline__ void to_host(uint64_t i, uint8_t* st, unsigned long long* marks, uint64_t* host_list,
                                        uint64_t host_cap) {
    st[i] = L_HOST;
    const unsigned long long q = atomicAdd(&marks[2], 1ull);
    if (q < host_cap) host_list[q] = i;
}

__device__ __forceinline__ void failed(uint64_t i, uint8_t code, uint8_t* st, unsigned long long* marks) {
    st[i] = code;
    atomicMin(&marks[1], (unsigned long long)i);
}

// One thread per line of the body: lines 0 .. L-1 end at nl[i]; line L (if
// the text does not end with a newline) ends at n.  A block's 256 lines are one
// range of the text, brought into shared memory by coalesced loads unless it is
// longer than kParseText.  Bound by instruction issue in the walks over a line's
// bytes: 24 MB (1M lines) take 123 us (from global memory 169, staged 159, and 123
// with the coordinates converted in integers); the host's arrays, made meanwhile,
// take as long.
constexpr uint32_t kParseText = 16384;
__global__ void __launch_bounds__(256) k_parse_lines(
    const uint8_t* __restrict__ buf, uint64_t n, const uint64_t* __restrict__ nl, uint64_t L, uint64_t lines,
    float* __restrict__ x, float* __restrict__ y, int32_t* __restrict__ raw, uint8_t* __restrict__ st,
    unsigned long long* __restrict__ marks, uint64_t* __restrict__ host_list, uint64_t host_cap) {
    __shared__ uint4 s_text[kParseText / 16];
    // marks[0]: first empty line, marks[1]: first malformed / id -1 line,
    // marks[2]: lines left to the host (their indices in host_list, unordered)
    const uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x, i = i0 + threadIdx.x;
    const uint64_t i1 = i0 + blockDim.x < lines ? i0 + blockDim.x : lines;
    const uint64_t first = (i0 == 0 ? 0 : nl[i0 - 1] + 1) & ~15ull;   // 16-byte aligned
    const uint64_t last = i1 - 1 < L ? nl[i1 - 1] : n;
    const bool staged = last - first <= kParseText;
    if (staged) {
        const uint32_t words = (uint32_t)((last - first + 15) / 16);
        for (uint32_t q = threadIdx.x; q < words; q += blockDim.x)
            s_text[q] = reinterpret_cast<const uint4*>(buf + first)[q];
        __syncthreads();
    }
    if (i >= lines) return;
    const uint64_t b = i == 0 ? 0 : nl[i - 1] + 1;
    uint64_t e = i < L ? nl[i] : n;
    const uint8_t* p = staged ? reinterpret_cast<const uint8_t*>(s_text) + (b - first) : buf + b;
    if (e > b && p[e - b - 1] == '\r') --e;
    if (e == b) {
        st[i] = L_EMPTY;
        atomicMin(&marks[0], (unsigned long long)i);
        return;
    }
    const uint8_t* pe = p + (e - b);
    const uint8_t *c1 = nullptr, *c2 = nullptr, *c3 = nullptr;
    for (const uint8_t* q = p; q < pe; ++q) {
        const uint8_t ch = *q;
        if (ch == '"' || ch == '\\') {   // the tokenizer's quotes and escapes: the host
            to_host(i, st, marks, host_list, host_cap);
            return;
        }
        if (ch == ',') {
            if (!c1) c1 = q;
            else if (!c2) c2 = q;
            else if (!c3) c3 = q;
        }
    }
    int32_t id = 0;
    float xv = 0.f, yv = 0.f;
    if (!c2 || parse_int_dev(p, c1, &id) != 0) {
        failed(i, L_BAD, st, marks);
        return;
    }
    const int fx = parse_float_dev(c1 + 1, c2, &xv);
    const int fy = parse_float_dev(c2 + 1, c3 ? c3 : pe, &yv);
    if (fx == 2 || fy == 2) {
        failed(i, L_BAD, st, marks);
        return;
    }
    if (fx == 1 || fy == 1) {   // the host decides (a float it rejects makes the line malformed)
        to_host(i, st, marks, host_list, host_cap);
        return;
    }
    if (id == -1) {
        failed(i, L_MINUS1, st, marks);
        return;
    }
    x[i] = xv;
    y[i] = yv;
    raw[i] = id;
    st[i] = L_OK;
}

// Group starts (the first point of every run of equal ids before the first empty
// line) with the byte range of their id field, for the feature names: out[2 q],
// out[2 q + 1], q < marks[3].  The bounds line (the one after the empty line)
// is marks[4] .. marks[5].
__global__ void k_group_starts(const int32_t* __restrict__ raw, uint64_t lines, const uint64_t* __restrict__ nl,
                               uint64_t L, uint64_t n, unsigned long long* __restrict__ marks,
                               uint64_t* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t empty = marks[0];
    if (i == 0 && empty < lines && empty + 1 < lines) {
        marks[4] = nl[empty] + 1;
        marks[5] = empty + 1 < L ? nl[empty + 1] : n;
    }
    if (i >= lines || i >= empty) return;
    if (i > 0 && raw[i] == raw[i - 1]) return;
    const unsigned long long k = atomicAdd(&marks[3], 1ull);
    out[2 * k] = i;
    out[2 * k + 1] = i == 0 ? 0 : nl[i - 1] + 1;
}

// Byte ranges [b, e) of the listed lines (a trailing '\r' kept; the host drops it).
__global__ void k_line_bounds(const uint64_t* __restrict__ idx, uint64_t m, const uint64_t* __restrict__ nl,
                              uint64_t L, uint64_t n, uint64_t* __restrict__ out) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m) return;
    const uint64_t i = idx[q];
    out[2 * q] = i == 0 ? 0 : nl[i - 1] + 1;
    out[2 * q + 1] = i < L ? nl[i] : n;
}

// Values of the lines parsed on the host, into the point arrays.
__global__ void k_scatter_points(const uint64_t* __restrict__ idx, const float* __restrict__ xs,
                                 const float* __restrict__ ys, const int32_t* __restrict__ ids, uint64_t m,
                                 float* __restrict__ x, float* __restrict__ y, int32_t* __restrict__ raw) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m) return;
    x[idx[q]] = xs[q];
    y[idx[q]] = ys[q];
    raw[idx[q]] = ids[q];
}

}  // namespace

colo_status parse_points_csv_device(cudaStream_t s, const char* path, HostPoints& hp, DevBuf<float>& dx,
                                    DevBuf<float>& dy, std::string& err) {
    // the file mapped (pages populated up front) and copied to the device from there
    struct Mapped {
        const char* p = nullptr;
        size_t n = 0;
        void* map = nullptr;
        bool ok = false;
        explicit Mapped(const char* path) {
            const int fd = ::open(path, O_RDONLY);
            if (fd < 0) return;
            struct stat st;
            if (::fstat(fd, &st) == 0) {
                n = (size_t)st.st_size;
                if (n == 0) {
                    ok = true;
                } else {
                    map = ::mmap(nullptr, n, PROT_READ, MAP_PRIVATE | MAP_POPULATE, fd, 0);
                    if (map != MAP_FAILED) {
                        p = static_cast<const char*>(map);
                        ok = true;
                    } else {
                        map = nullptr;
                    }
                }
            }
            ::close(fd);
        }
        ~Mapped() {
            if (map) ::munmap(map, n);
        }
    } file(path);
    if (!file.ok) {
        err = std::string("cannot read dataset: ") + path;
        return COLO_ERR_IO;
    }
    const char* beg = file.p;
    const char* end = beg + file.n;
    // the count line, on the host
    const char* nl0 = file.n == 0 ? nullptr : (const char*)std::memchr(beg, '\n', file.n);
    const char* le0 = nl0 ? nl0 : end;
    if (le0 > beg && le0[-1] == '\r') --le0;
    long N = 0;
    if (file.n == 0 || !csv_parse_count(beg, le0, &N)) {
        err = "dataset: first line must hold the point count";
        return COLO_ERR_PARSE;
    }
    const char* body = nl0 ? nl0 + 1 : end;
    const uint64_t nb = (uint64_t)(end - body);
    hp.clear();
    // the text on the device, and its line ends: into room for lines of points, and once more
    // when there are more (the kernel counts them all)
    DevBuf<uint8_t> dbuf;
    dbuf.alloc((nb + 15) / 16 * 16 + 16, s);
    if (nb) COLO_CUDA(cudaMemcpyAsync(dbuf.get(), body, nb, cudaMemcpyHostToDevice, s));
    const uint64_t tiles = (nb + kNlTile - 1) / kNlTile;
    DevBuf<unsigned long long> words;
    DevBuf<uint64_t> dnl;
    uint64_t L = 0, cap = nb / kMinLine + 64;
    // the host's arrays are made while the device works (at most a line of the text per point)
    const uint64_t room = std::min<uint64_t>(N > 0 ? (uint64_t)N : 0u, nb / kMinLine + 1);
    for (bool again = tiles > 0; again;) {
        dnl.alloc(cap, s);
        words.alloc(tiles + 1, s);
        words.zero(s);
        {
            KScope ks("csv_lines");
            k_line_ends<<<(unsigned)tiles, kNlThreads, 0, s>>>(
                dbuf.get(), nb, words.get(), reinterpret_cast<uint32_t*>(words.get() + tiles), dnl.get(), cap);
            COLO_LAUNCH_CHECK();
            count_launch();
        }
        hp.x.resize(room);
        COLO_CUDA(cudaMemcpyAsync(&L, words.get() + tiles - 1, 8, cudaMemcpyDeviceToHost, s));
        stream_wait(s);
        L &= kScanVal;
        again = L > cap;
        cap = L;
    }
    // a last line without its newline counts too (std::getline)
    const uint64_t lines = L + (nb > 0 && end[-1] != '\n' ? 1 : 0);
    // every line parsed on the device, then the groups of the lines before the first empty one
    DevBuf<float> px, py;
    DevBuf<int32_t> praw;
    DevBuf<uint8_t> pst;
    DevBuf<uint64_t> hlist;
    constexpr uint64_t kMarks = 6, kFirstGroups = 256;
    const uint64_t host_cap = std::max<uint64_t>(1024, lines / 64);
    DevBuf<unsigned long long> marks;   // the marks, then the groups
    marks.alloc(kMarks + 2 * std::max(lines, kFirstGroups), s);
    hlist.alloc(host_cap, s);
    {
        const unsigned long long init[kMarks] = {~0ull, ~0ull, 0ull, 0ull, 0ull, 0ull};
        COLO_CUDA(cudaMemcpyAsync(marks.get(), init, sizeof(init), cudaMemcpyHostToDevice, s));
    }
    uint64_t* const groups = reinterpret_cast<uint64_t*>(marks.get() + kMarks);
    px.alloc(lines ? lines : 1, s);
    py.alloc(lines ? lines : 1, s);
    praw.alloc(lines ? lines : 1, s);
    pst.alloc(lines ? lines : 1, s);
    auto list_groups = [&] {
        KScope ks("csv_groups");
        k_group_starts<<<(unsigned)((lines + 255) / 256), 256, 0, s>>>(praw.get(), lines, dnl.get(), L, nb,
                                                                      marks.get(), groups);
        COLO_LAUNCH_CHECK();
        count_launch();
    };
    if (lines) {
        {
            KScope ks("csv_parse");
            k_parse_lines<<<(unsigned)((lines + 255) / 256), 256, 0, s>>>(dbuf.get(), nb, dnl.get(), L, lines,
                                                                         px.get(), py.get(), praw.get(), pst.get(),
                                                                         marks.get(), hlist.get(), host_cap);
            COLO_LAUNCH_CHECK();
            count_launch();
        }
        list_groups();
    }
    hp.y.resize(room);
    hp.raw.resize(room);
    std::vector<unsigned long long> hm(kMarks + 2 * kFirstGroups);
    auto read_marks = [&] {
        COLO_CUDA(cudaMemcpyAsync(hm.data(), marks.get(), hm.size() * 8, cudaMemcpyDeviceToHost, s));
        stream_wait(s);
    };
    read_marks();
    const unsigned long long first_empty = hm[0];
    const uint64_t np = first_empty < lines ? first_empty : lines;   // point lines before the empty line
    // the first failing device line before the empty line, and its kind
    const uint64_t first_bad = hm[1] < np ? hm[1] : np;
    uint8_t bad_kind = L_BAD;
    if (first_bad < np) COLO_CUDA(cudaMemcpy(&bad_kind, pst.get() + first_bad, 1, cudaMemcpyDeviceToHost));
    // lines the host reads: the listed ones before the first device failure, and the bounds line
    std::vector<uint64_t> want;
    if (hm[2] > host_cap) {   // more than the list holds: find them from the statuses
        std::vector<uint8_t> hst(np);
        if (np) COLO_CUDA(cudaMemcpy(hst.data(), pst.get(), np, cudaMemcpyDeviceToHost));
        for (uint64_t i = 0; i < first_bad; ++i)
            if (hst[i] == L_HOST) want.push_back(i);
    } else if (hm[2]) {
        std::vector<uint64_t> hl(hm[2]);
        COLO_CUDA(cudaMemcpy(hl.data(), hlist.get(), hm[2] * 8, cudaMemcpyDeviceToHost));
        for (uint64_t i : hl)
            if (i < first_bad) want.push_back(i);
        std::sort(want.begin(), want.end());
    }
    const bool has_bounds = first_empty < lines && first_empty + 1 < lines;
    std::vector<uint64_t> rng(2 * want.size());
    if (!want.empty()) {
        DevBuf<uint64_t> didx, drng;
        didx.alloc(want.size(), s);
        drng.alloc(2 * want.size(), s);
        COLO_CUDA(cudaMemcpyAsync(didx.get(), want.data(), want.size() * 8, cudaMemcpyHostToDevice, s));
        k_line_bounds<<<(unsigned)((want.size() + 255) / 256), 256, 0, s>>>(didx.get(), want.size(), dnl.get(), L,
                                                                           nb, drng.get());
        COLO_LAUNCH_CHECK();
        count_launch();
        COLO_CUDA(cudaMemcpyAsync(rng.data(), drng.get(), rng.size() * 8, cudaMemcpyDeviceToHost, s));
        COLO_CUDA(cudaStreamSynchronize(s));
    }
    auto line_at = [&](size_t q, const char** lb, const char** lend) {
        *lb = body + rng[2 * q];
        *lend = body + rng[2 * q + 1];
        if (*lend > *lb && (*lend)[-1] == '\r') --*lend;
    };
    // host lines in order: the first failing line, device or host, is the one the serial reader names
    const size_t nhost = want.size();
    std::vector<std::pair<uint64_t, std::string>> host_tokens;
    std::vector<uint64_t> hidx;
    std::vector<float> hxv, hyv;
    std::vector<int32_t> hrv;
    for (size_t q = 0; q < nhost; ++q) {
        const uint64_t i = want[q];
        const char *lb, *lend;
        line_at(q, &lb, &lend);
        int32_t id;
        float xv, yv;
        bool m1 = false;
        std::string tok;
        if (!csv_parse_line(lb, lend, &id, &xv, &yv, &m1, &tok)) {
            err = m1 ? "dataset: feature id -1 is the reference's 'no feature yet' marker (line " +
                           std::to_string(i + 2) + ")"
                     : "dataset: malformed point line " + std::to_string(i + 2);
            return COLO_ERR_PARSE;
        }
        hidx.push_back(i);
        hxv.push_back(xv);
        hyv.push_back(yv);
        hrv.push_back(id);
        host_tokens.emplace_back(i, std::move(tok));
    }
    if (first_bad < np) {
        err = bad_kind == L_MINUS1 ? "dataset: feature id -1 is the reference's 'no feature yet' marker (line " +
                                               std::to_string(first_bad + 2) + ")"
                                         : "dataset: malformed point line " + std::to_string(first_bad + 2);
        return COLO_ERR_PARSE;
    }
    if ((long)np != N) {
        err = "dataset: count line says " + std::to_string(N) + " points, found " + std::to_string(np);
        return COLO_ERR_PARSE;
    }
    if (!has_bounds) {
        err = "dataset: bounds line missing";
        return COLO_ERR_PARSE;
    }
    {
        const char *lb = body + hm[4], *lend = body + hm[5];
        if (lend > lb && lend[-1] == '\r') --lend;
        if (!csv_parse_bounds(lb, lend, hp.bounds)) {
            err = "dataset: bounds line must be minX,minY,maxX,maxY";
            return COLO_ERR_PARSE;
        }
    }
    // the host's values into the device arrays
    if (!hidx.empty()) {
        const uint64_t m = hidx.size();
        DevBuf<uint64_t> di;
        DevBuf<float> dxs, dys;
        DevBuf<int32_t> dis;
        di.alloc(m, s);
        dxs.alloc(m, s);
        dys.alloc(m, s);
        dis.alloc(m, s);
        COLO_CUDA(cudaMemcpyAsync(di.get(), hidx.data(), m * 8, cudaMemcpyHostToDevice, s));
        COLO_CUDA(cudaMemcpyAsync(dxs.get(), hxv.data(), m * 4, cudaMemcpyHostToDevice, s));
        COLO_CUDA(cudaMemcpyAsync(dys.get(), hyv.data(), m * 4, cudaMemcpyHostToDevice, s));
        COLO_CUDA(cudaMemcpyAsync(dis.get(), hrv.data(), m * 4, cudaMemcpyHostToDevice, s));
        k_scatter_points<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(di.get(), dxs.get(), dys.get(), dis.get(), m,
                                                                    px.get(), py.get(), praw.get());
        COLO_LAUNCH_CHECK();
        count_launch();
        COLO_CUDA(cudaMemsetAsync(marks.get() + 3, 0, 8, s));
        list_groups();
        read_marks();   // the host vectors above are about to go
    }
    const uint64_t G = hm[3];
    hp.x.resize(np);
    hp.y.resize(np);
    hp.raw.resize(np);
    if (np) {
        COLO_CUDA(cudaMemcpyAsync(hp.x.data(), px.get(), np * 4, cudaMemcpyDeviceToHost, s));
        COLO_CUDA(cudaMemcpyAsync(hp.y.data(), py.get(), np * 4, cudaMemcpyDeviceToHost, s));
        COLO_CUDA(cudaMemcpyAsync(hp.raw.data(), praw.get(), np * 4, cudaMemcpyDeviceToHost, s));
    }
    hm.resize(kMarks + 2 * std::max(G, kFirstGroups));
    if (G > kFirstGroups) COLO_CUDA(cudaMemcpyAsync(hm.data() + kMarks, groups, 2 * G * 8, cudaMemcpyDeviceToHost, s));
    COLO_CUDA(cudaStreamSynchronize(s));
    const unsigned long long* g = hm.data() + kMarks;
    std::vector<std::pair<uint64_t, uint64_t>> starts(G);
    for (uint64_t q = 0; q < G; ++q) starts[q] = {g[2 * q], g[2 * q + 1]};
    std::sort(starts.begin(), starts.end());
    size_t hq = 0;
    hp.tokens.reserve(G);
    for (const auto& st : starts) {
        const uint64_t i = st.first;
        while (hq < host_tokens.size() && host_tokens[hq].first < i) ++hq;
        if (hq < host_tokens.size() && host_tokens[hq].first == i) {
            hp.tokens.emplace_back(i, host_tokens[hq].second);   // the tokenizer's unescaped field
            continue;
        }
        const char* lb = body + st.second;   // a device-parsed line: plain text up to the first comma
        const char* c1 = (const char*)std::memchr(lb, ',', (size_t)(end - lb));
        hp.tokens.emplace_back(i, std::string(lb, c1 ? c1 : lb));
    }
    hp.tokens_complete = true;
    dx = std::move(px);
    dy = std::move(py);
    return COLO_OK;
}

}  // namespace colo
