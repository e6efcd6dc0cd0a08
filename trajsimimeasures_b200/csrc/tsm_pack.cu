// Host side of the paired call on padded host arrays: the valid points of a
// batch, translated and rounded to float32, packed into one staging buffer with
// the offsets and lengths that tsm_pairs takes, so that a call is one pass over
// the points that count and one upload.
//
// Bound by the host's memory (16 bytes read and 8 written a point; 2.2 ms, 48
// GB/s, for 20,000 pairs).  Measured on the host of a B200, pairs of 20..200
// float64 points padded to 200: 512 of them 197 us as one array operation over
// the padded width per side, 113 us here; 64 of them 8 us.
#include <emmintrin.h>

#include <cmath>
#include <cstring>
#include <thread>
#include <type_traits>
#include <vector>

#include "tsm.h"

int tsm_internal_fail(int code, const char* msg);

namespace {

struct Side {
    const unsigned char* base;
    int64_t traj, pt;  // byte strides
    const int64_t* len;
    int64_t* off;
    int32_t* len32;
};

template <class T>
void pack_rows(const Side& s, int64_t k0, int64_t k1, const double* origin, bool per_pair, float* dst) {
    for (int64_t k = k0; k < k1; ++k) {
        const int64_t n = s.len[k];
        const unsigned char* p = s.base + k * s.traj;
        float* d = dst + 2 * s.off[k];
        if (!origin) {
            if (std::is_same<T, float>::value && s.pt == 8) {  // as they are
                if (n > 0) std::memcpy(d, p, (size_t)(8 * n));
                continue;
            }
            for (int64_t i = 0; i < n; ++i) {
                const T* q = reinterpret_cast<const T*>(p + i * s.pt);
                d[2 * i] = (float)q[0];
                d[2 * i + 1] = (float)q[1];
            }
            continue;
        }
        const double ox = origin[per_pair ? 2 * k : 0], oy = origin[per_pair ? 2 * k + 1 : 1];
        if (std::is_same<T, double>::value) {  // a point's two coordinates at a time, whatever lies between points
            const __m128d o2 = _mm_set_pd(oy, ox);
            for (int64_t i = 0; i < n; ++i) {
                const __m128d v = _mm_loadu_pd(reinterpret_cast<const double*>(p + i * s.pt));
                _mm_storel_pi(reinterpret_cast<__m64*>(d + 2 * i), _mm_cvtpd_ps(_mm_sub_pd(v, o2)));
            }
            continue;
        }
        if (s.pt == 2 * (int64_t)sizeof(T)) {  // contiguous points
            const T* q = reinterpret_cast<const T*>(p);
            for (int64_t i = 0; i < n; ++i) {
                d[2 * i] = (float)((double)q[2 * i] - ox);
                d[2 * i + 1] = (float)((double)q[2 * i + 1] - oy);
            }
        } else {
            for (int64_t i = 0; i < n; ++i) {
                const T* q = reinterpret_cast<const T*>(p + i * s.pt);
                d[2 * i] = (float)((double)q[0] - ox);
                d[2 * i + 1] = (float)((double)q[1] - oy);
            }
        }
    }
}

template <class T>
void first_point(const Side& s, int64_t k, double* o) {
    const T* q = reinterpret_cast<const T*>(s.base + k * s.traj);
    o[0] = (double)(float)(double)q[0];
    o[1] = (double)(float)(double)q[1];
}

template <class T>
void pack_all(const Side& a, const Side& b, int64_t n, int mode, const double* origin, float* dst, int64_t total) {
    std::vector<double> own;
    if (mode == TSM_ORIGIN_PER_PAIR) {
        own.assign((size_t)(2 * n), 0.0);
        for (int64_t k = 0; k < n; ++k) {
            double* o = own.data() + 2 * k;
            if (a.len[k] > 0) first_point<T>(a, k, o);
            else if (b.len[k] > 0) first_point<T>(b, k, o);
            if (!std::isfinite(o[0]) || !std::isfinite(o[1])) o[0] = o[1] = 0.0;
        }
        origin = own.data();
    }
    const double* o = mode == TSM_ORIGIN_NONE ? nullptr : origin;
    const bool per_pair = mode == TSM_ORIGIN_PER_PAIR;
    auto part = [&](int64_t k0, int64_t k1) {
        pack_rows<T>(a, k0, k1, o, per_pair, dst);
        pack_rows<T>(b, k0, k1, o, per_pair, dst);
    };
    // Threads only where the pass is long: started on idle cores, they cost a call
    // more than the pass they share.  A call in one thread / in threads of
    // 262,144 / of 524,288 / of 98,304 points (float64 pairs of 20..200): 1,000
    // pairs 0.49 ms / - / - / 0.54, 4,096 (0.9 million points) 1.34 / 1.20 / - /
    // 1.54 (float32 1.11 / 1.21 / - / 1.74), 6,000 (float32) 1.55 / 1.87 / 1.48,
    // 20,000 12.5 / 5.1 / 5.0.  Points that are not back to back (a slice of wider
    // rows) are bound by one core's loads sooner: 40 bytes apart, 1,500 pairs 0.83 ms
    // in one thread, 0.73 in threads of 131,072, 4,096 1.96 / 1.31.  (Array operations
    // over the padded width, in a pool that is always there: 0.62 and 1.32; 1,000
    // pairs 0.50, here in one thread 0.62.)
    const bool dense = a.pt == 2 * (int64_t)sizeof(T) && b.pt == a.pt;
    int64_t nt = total / (dense ? 524288 : 131072);
    const int64_t hw = (int64_t)std::thread::hardware_concurrency();
    if (nt > 8) nt = 8;
    if (nt > hw) nt = hw;
    if (nt < 2) return part(0, n);
    std::vector<std::thread> th;
    th.reserve((size_t)nt);
    int64_t done = 0;  // pairs handed to threads (the calling one takes what is left)
    try {
        for (int64_t t = 0; t + 1 < nt; ++t) {
            const int64_t k1 = n * (t + 1) / nt;
            th.emplace_back(part, done, k1);
            done = k1;
        }
    } catch (...) {  // no more threads to be had
    }
    part(done, n);
    for (auto& t : th) t.join();
}

}  // namespace

extern "C" {

int tsm_pack_pairs(const void* t1, int64_t traj_stride1, int64_t pt_stride1, const int64_t* len1, const void* t2,
                   int64_t traj_stride2, int64_t pt_stride2, const int64_t* len2, int64_t n, int32_t type,
                   int32_t origin_mode, const double* origin, int64_t* off_a, int64_t* off_b, int32_t* len_a,
                   int32_t* len_b, float* pts, int64_t max_points) {
    if (n < 0) return tsm_internal_fail(TSM_EINVAL, "tsm_pack_pairs: n < 0");
    if (n == 0) return TSM_OK;
    if (!t1 || !t2 || !len1 || !len2 || !off_a || !off_b || !len_a || !len_b || !pts)
        return tsm_internal_fail(TSM_EINVAL, "tsm_pack_pairs: null pointer");
    if (origin_mode < TSM_ORIGIN_NONE || origin_mode > TSM_ORIGIN_ONE || (origin_mode == TSM_ORIGIN_ONE && !origin))
        return tsm_internal_fail(TSM_EINVAL, "tsm_pack_pairs: bad origin");
    if (type < TSM_F32 || type > TSM_I64) return tsm_internal_fail(TSM_EINVAL, "tsm_pack_pairs: unknown type");
    try {
        int64_t at = 0;
        for (int side = 0; side < 2; ++side) {
            const int64_t* len = side ? len2 : len1;
            int64_t* off = side ? off_b : off_a;
            int32_t* l32 = side ? len_b : len_a;
            for (int64_t k = 0; k < n; ++k) {
                if (len[k] < 0 || len[k] > max_points - at)
                    return tsm_internal_fail(TSM_EINVAL, "tsm_pack_pairs: lengths negative or beyond max_points");
                off[k] = at;
                l32[k] = (int32_t)len[k];
                at += len[k];
            }
        }
        const Side a{static_cast<const unsigned char*>(t1), traj_stride1, pt_stride1, len1, off_a, len_a};
        const Side b{static_cast<const unsigned char*>(t2), traj_stride2, pt_stride2, len2, off_b, len_b};
        switch (type) {
            case TSM_F32: pack_all<float>(a, b, n, origin_mode, origin, pts, at); break;
            case TSM_F64: pack_all<double>(a, b, n, origin_mode, origin, pts, at); break;
            case TSM_I32: pack_all<int32_t>(a, b, n, origin_mode, origin, pts, at); break;
            default: pack_all<int64_t>(a, b, n, origin_mode, origin, pts, at);
        }
    } catch (...) {
        return tsm_internal_fail(TSM_EINVAL, "tsm_pack_pairs: out of memory");
    }
    return TSM_OK;
}

}  // extern "C"
