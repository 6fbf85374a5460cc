// Unfolding of QCMaquis RDM label/value lists into the dense arrays of the
// path: src/rdm_utils.F90:236-464 permute_4rdm (into the packed 4-RDM
// ro4(W,n,n,n,n) of one state) and :470-511 permute_3rdm (into a 3-RDM
// (n,n,n,n,n,n) of one state or root pair), as hdf5_read_rdm_from_resfile
// (src/rdm_utils.F90:193-226) applies them: labels + 1, one call per entry in
// file order, every image an assignment (a later entry overwrites an earlier
// one on the same element; within one entry a later image overwrites an
// earlier one).
//
// GPU form: pass 1, a thread per entry, claims each destination element with the
// key (entry, image, weight) + 1 by atomicMax; pass 2, a thread per destination
// element, writes the value of the entry whose key won.  The result is the one of
// the sequential loop, bit for bit, independent of thread order.
//
// Bound by the label reads of pass 1 (32 bytes an entry) and the element pass.
// The weight travels in the key and the elements are written in their own order, so
// the labels are read once and the stores are coalesced; the images are addressed as
// they are enumerated (a table of them lived in local memory).  Keys of 32 bits hold
// 2^26 entries and halve the claim array; longer lists take 64 bits.  CAS(9), all
// 1.6 million entries, with the host call: 165 -> 72 us.
#include "eexx.cuh"
#include "nvpt2_internal.h"

namespace nvpt {

namespace {

constexpr double kRdmThresh = 1.0e-12;  // src/rdm_utils.F90:241 / :479

// The image table of permute_4rdm for one label (1-based indices), in the
// reference's order: put(a, b, c, d, w) for each of the 0..12 images, (a, b, c, d)
// the permuted (m, n, o, p); w 0: val, 1: -val/2, 2: -2 val.
template <class F>
__device__ __forceinline__ void images4(int i, int j, int k, int l, int m, int n, int o, int p, F put) {
    const int V = 0, H = 1, T = 2;
    if (i == j && k == l) {  // case 1
        if (m == n && o == p) {
            put(m, n, o, o, V); put(o, o, m, m, V);
            put(m, o, o, m, H); put(m, o, m, o, H); put(o, m, m, o, H); put(o, m, o, m, H);
        } else if (m == n && o != p) {
            put(m, n, o, p, V); put(m, m, p, o, V); put(o, p, m, m, V); put(p, o, m, m, V);
            put(o, m, m, p, H); put(o, m, p, m, H); put(p, m, m, o, H); put(p, m, o, m, H);
            put(m, o, p, m, H); put(m, p, o, m, H); put(m, p, m, o, H); put(m, o, m, p, H);
        } else if (m != n && o == p) {
            put(m, n, o, p, V); put(n, m, o, o, V); put(o, o, m, n, V); put(o, o, n, m, V);
            put(m, o, o, n, H); put(n, o, o, m, H); put(o, m, o, n, H); put(o, n, o, m, H);
            put(o, m, n, o, H); put(o, n, m, o, H); put(m, o, n, o, H); put(n, o, m, o, H);
        } else {  // m != n, o != p
            if (n == o) {
                put(m, n, o, p, V);
                put(n, n, m, p, T); put(n, n, p, m, T); put(m, p, n, n, T); put(p, m, n, n, T);
                put(p, n, n, m, V); put(p, n, m, n, V); put(m, n, p, n, V); put(n, p, m, n, V);
                put(n, m, p, n, V); put(n, m, n, p, V); put(n, p, n, m, V);
            } else {  // both remaining branches of the reference write the same eight images
                put(m, n, o, p, V); put(m, n, p, o, V); put(n, m, p, o, V); put(n, m, o, p, V);
                put(o, p, m, n, V); put(o, p, n, m, V); put(p, o, n, m, V); put(p, o, m, n, V);
            }
        }
    } else if (i == j && k != l) {  // case 2
        if (m == n && o == p) {
            put(m, n, o, p, V); put(o, o, m, m, V);
            put(m, o, o, m, H); put(o, m, m, o, H); put(o, m, o, m, H); put(m, o, m, o, H);
        }
        if (m == n && o != p) {
            put(m, n, o, p, V);
            put(m, o, m, p, H); put(m, p, o, m, H); put(o, m, m, p, H); put(p, m, o, m, H);
        }
        if (m != n && o == p) {
            put(m, n, o, p, V); put(n, m, o, o, V);
        }
        if (m != n && n != o && o != p && m != p) {
            put(m, n, o, p, V); put(n, m, o, p, V);
        }
    } else if (i != j && j == k && k != l) {  // case 3
        if (m == n && o == p) {
            put(m, n, o, p, V); put(o, o, m, m, V); put(o, m, o, m, V); put(m, o, m, o, V);
            put(m, o, o, m, T); put(o, m, m, o, T);
        }
        if (m != n && o == p) {
            put(m, n, o, p, V); put(o, o, m, n, V); put(o, m, o, n, V); put(m, o, n, o, V);
            put(m, o, o, n, T);
        }
        if (m != n && o != p && m == p) {
            put(m, n, o, p, V); put(m, o, n, m, V);
        }
        if (m != n && n != o && o != p && m != p) {
            put(m, n, o, p, V); put(m, o, n, p, V);
        }
    } else if (i != j && k == l) {  // case 4
        if (m == n && o == p) {
            put(m, n, o, p, V); put(o, o, m, m, V);
            put(m, o, o, m, H); put(o, m, m, o, H); put(o, m, o, m, H); put(m, o, m, o, H);
        }
        if (m == n && o != p) {
            put(m, n, o, p, V); put(m, m, p, o, V);
        }
        if (m != n && o == p) {
            put(m, n, o, p, V);
            put(m, o, n, o, H); put(m, o, o, n, H); put(o, n, o, m, H); put(o, n, m, o, H);
        }
        if (m != n && n != o && o != p && m != p) {
            put(m, n, o, p, V); put(m, n, p, o, V);
        }
    } else if (i != j && k != l && j != k) {  // case 5
        if ((m == o && n == p) || (m == p && n == o)) {
            put(m, n, o, p, V); put(n, m, p, o, V);
        } else if (m == n && o == p) {
            put(m, n, o, p, V); put(o, o, m, m, V);
        } else {
            put(m, n, o, p, V);
        }
    }
}

__device__ __forceinline__ double weighted(double v, int w) {
    return w == 0 ? v : (w == 1 ? v * (-0.5) : v * (-2.0));
}

__device__ __forceinline__ bool label_ok(const int *L, int k, int n) {
    for (int q = 0; q < k; ++q)
        if (L[q] < 0 || L[q] >= n) return false;
    return true;
}

// Keys: entry (the high bits), image (4 bits), weight (2 bits), plus one; 0 = unclaimed.
constexpr int kKeyBits = 6;

// VEC: the labels are 16-byte aligned.
template <class Key, bool VEC>
__global__ void __launch_bounds__(256) k_claim4(const int32_t *__restrict__ lab, const double *__restrict__ val, ll ne,
                                                int n, ll W, Key *owner, int *bad) {
    const ll e = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    int q[8];
    if (VEC) {
        const int4 a = reinterpret_cast<const int4 *>(lab)[2 * e], b = reinterpret_cast<const int4 *>(lab)[2 * e + 1];
        q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
        q[4] = b.x; q[5] = b.y; q[6] = b.z; q[7] = b.w;
    } else {
#pragma unroll
        for (int t = 0; t < 8; ++t) q[t] = lab[8 * e + t];
    }
    if (!label_ok(q, 8, n)) {
        atomicExch(bad, 1);
        return;
    }
    if (fabs(val[e]) < kRdmThresh) return;
    Key *at = owner + normind4(q[0] + 1, q[1] + 1, q[2] + 1, q[3] + 1) - 1;
    Key key = ((Key)e << kKeyBits) + 1;
    images4(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], [&](int a, int b, int c, int d, int w) {
        atomicMax(at + W * (a + (ll)n * (b + (ll)n * (c + (ll)n * d))), key + w);
        key += 4;
    });
}

// crowded: more than kCrowded entries an element.  A file holds an element once, but
// nothing says so, and the entries of such a list fight for the same claims, twelve a
// thread: a claim that a later entry has won is then left alone (n = 3, 100 000 entries,
// the host call: 195 -> 160 us).  Elsewhere the load ahead of each claim is not free.
constexpr int kCrowded = 16;
template <class Key>
__global__ void __launch_bounds__(256) k_claim3(const int32_t *__restrict__ lab, const double *__restrict__ val, ll ne,
                                                int n, int trans, Key *owner, int *bad, bool crowded) {
    const ll e = (ll)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    int q[6];
#pragma unroll
    for (int t = 0; t < 6; ++t) q[t] = lab[6 * e + t];
    if (!label_ok(q, 6, n)) {
        atomicExch(bad, 1);
        return;
    }
    if (fabs(val[e]) < kRdmThresh) return;
    const int i = q[0], j = q[1], k = q[2], l = q[3], m = q[4], nn = q[5];
    if (i == j && i == k) return;
    if (l == m && l == nn) return;
    // every image of an entry has the same value, and the value's sign is trans's
    // (src/rdm_utils.F90:486): the images need no order
    const Key key = ((Key)e << kKeyBits) + 1;
    auto put = [&](int a, int b, int c, int d, int f, int g) {
        Key *at = owner + (a + (ll)n * (b + (ll)n * (c + (ll)n * (d + (ll)n * (f + (ll)n * g)))));
        if (!crowded || *(volatile Key *)at < key) atomicMax(at, key);
    };
    put(i, j, k, l, m, nn); put(i, k, j, l, nn, m); put(j, i, k, m, l, nn);
    put(j, k, i, m, nn, l); put(k, i, j, nn, l, m); put(k, j, i, nn, m, l);
    if (trans) return;
    put(l, m, nn, i, j, k); put(l, nn, m, i, k, j); put(m, l, nn, j, i, k);
    put(m, nn, l, j, k, i); put(nn, l, m, k, i, j); put(nn, m, l, k, j, i);
}

// dst[at * ld] = the value of the claim on `at`, R elements a thread.
template <class Key>
__global__ void __launch_bounds__(256) k_assign(const Key *__restrict__ owner, ll slots, const double *__restrict__ val,
                                                bool negate, double *dst, ll ld) {
    constexpr int R = 4;
    const ll at0 = (ll)blockIdx.x * (256 * R) + threadIdx.x;
    Key key[R];
    double v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const ll at = at0 + 256 * r;
        key[r] = at < slots ? owner[at] : 0;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = key[r] ? val[(key[r] - 1) >> kKeyBits] : 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (key[r]) {
            const double x = weighted(v[r], (int)((key[r] - 1) & 3));
            dst[(at0 + 256 * r) * ld] = negate ? -x : x;
        }
}

template <class Key>
int unfold4(const int32_t *labels, const double *values, ll ne, int n, ll slots, double *ro4, Key *owner, int *bad,
            cudaStream_t st) {
    const ll W = (ll)n * (n + 1) * (n + 2) * (n + 3) / 24;
    const unsigned g = (unsigned)((ne + 255) / 256);
    if ((uintptr_t)labels % 16 == 0) k_claim4<Key, true><<<g, 256, 0, st>>>(labels, values, ne, n, W, owner, bad);
    else k_claim4<Key, false><<<g, 256, 0, st>>>(labels, values, ne, n, W, owner, bad);
    k_assign<Key><<<(unsigned)((slots + 1023) / 1024), 256, 0, st>>>(owner, slots, values, false, ro4, 1);
    g_launches.fetch_add(2, std::memory_order_relaxed);
    return 0;
}

template <class Key>
int unfold3(const int32_t *labels, const double *values, ll ne, int n, ll slots, double *r3, ll ld, bool trans,
            Key *owner, int *bad, cudaStream_t st) {
    k_claim3<Key><<<(unsigned)((ne + 255) / 256), 256, 0, st>>>(labels, values, ne, n, trans ? 1 : 0, owner, bad,
                                                                       ne / kCrowded > slots);
    k_assign<Key><<<(unsigned)((slots + 1023) / 1024), 256, 0, st>>>(owner, slots, values, !trans, r3, ld);
    g_launches.fetch_add(2, std::memory_order_relaxed);
    return 0;
}

}  // namespace

size_t unfold_scratch(int which, int n, long long nentries) {
    const ll slots = (which == 4 ? (ll)n * (n + 1) * (n + 2) * (n + 3) / 24 : (ll)n * n) * n * n * n * n;
    return (size_t)slots * (nentries < (1ll << (32 - kKeyBits)) ? 4 : 8);
}

int launch_unfold4(const int32_t *labels, const double *values, long long nentries, int n, double *ro4, void *owner,
                   int *bad, cudaStream_t st) {
    const size_t bytes = unfold_scratch(4, n, nentries);
    const ll slots = (ll)n * (n + 1) * (n + 2) * (n + 3) / 24 * n * n * n * n;
    if (nentries == 0) return 0;
    if (cudaMemsetAsync(owner, 0, bytes, st) != cudaSuccess) return 1;
    if (bytes == (size_t)slots * 4) return unfold4(labels, values, nentries, n, slots, ro4, (unsigned *)owner, bad, st);
    return unfold4(labels, values, nentries, n, slots, ro4, (unsigned long long *)owner, bad, st);
}

int launch_unfold3(const int32_t *labels, const double *values, long long nentries, int n, double *rdm3, long long ld,
                   bool trans, void *owner, int *bad, cudaStream_t st) {
    const size_t bytes = unfold_scratch(3, n, nentries);
    const ll slots = (ll)n * n * n * n * n * n;
    if (nentries == 0) return 0;
    if (cudaMemsetAsync(owner, 0, bytes, st) != cudaSuccess) return 1;
    if (bytes == (size_t)slots * 4)
        return unfold3(labels, values, nentries, n, slots, rdm3, ld, trans, (unsigned *)owner, bad, st);
    return unfold3(labels, values, nentries, n, slots, rdm3, ld, trans, (unsigned long long *)owner, bad, st);
}

}  // namespace nvpt
