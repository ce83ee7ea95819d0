// capi.cu -- the C ABI of libphylogenetics.so.
//
// The first three symbols are the drop-in boundary: same names, argument order
// and meaning as the reference's JNA interface
// (src/main/java/nl/esciencecenter/phylogenetics_analysis/Bindings.java:17-45)
// and its C definitions (phylogenetics/src/main/cpp/native.cu:705-780):
//   * the caller owns every device buffer and the stream; the library uses the
//     caller's current context and never allocates, frees or selects a device;
//   * calls are synchronous (the stream is synchronised before returning);
//   * the return value is a cudaError_t code, 0 on success, with a message on
//     stderr for argument errors (cudaErrorUnknown, as the reference).
// compareCompositionVectors returns int (the Java binding's type); the
// reference's C definition says double and returns the code converted to
// double, which a caller binding int reads from the wrong register.
//
// The remaining symbols (phylo*) are new: batched construction into an arena,
// the window index and the pair-engine launches used by the batched and
// serving paths.  They follow the same conventions but are asynchronous unless
// stated.
#include <string.h>

#include <vector>

#include "../../include/phylogenetics.h"
#include "allpairs.cuh"
#include "compare.cuh"
#include "cv_build.cuh"
#include "hostctx.cuh"
#include "postings.cuh"
#include "rank.cuh"
#include "scan.cuh"

using namespace phylo;

namespace {

int parse_alphabet(const char *alphabet) {
    if (!alphabet) return -1;
    if (strcmp(alphabet, "DNA") == 0) return ALPHA_DNA;
    if (strcmp(alphabet, "protein") == 0) return ALPHA_PROTEIN;
    return -1;
}

// Candidate capacity reserved for one proteome of at most max_size entries.
// Candidates = entries + the slots whose alpha is exactly zero; they can never
// exceed the dense slot count A^K.
uint64_t single_cand_cap(const BuildGeometry &g, uint64_t max_size) {
    uint64_t cap = 2 * max_size + (1u << 20);
    const uint64_t dense = (uint64_t)g.T1 * g.A;
    return cap < dense ? cap : dense;
}

// arena offsets: vec_off[p] = base + sum of nnz rounded up to 4 entries; the padding
// entries after each vector get key 0xffffffff, value 0.  One CTA.
constexpr int AO_THREADS = 256;
__global__ void __launch_bounds__(AO_THREADS) k_arena_offsets(const uint64_t *nnz, int B,
                                                              uint64_t base, uint64_t *vec_off,
                                                              uint64_t *dst_base, uint64_t *dst_cap,
                                                              uint32_t *keys, float *vals) {
    __shared__ uint64_t sw[AO_THREADS / 32 + 1];
    uint64_t run = base;
    for (int p0 = 0; p0 < B; p0 += AO_THREADS) {
        const int p = p0 + threadIdx.x;
        const uint64_t n = p < B ? nnz[p] : 0, len = (n + 3) & ~(uint64_t)3;
        uint64_t tot;
        const uint64_t off = run + block_excl_scan_u64<AO_THREADS>(len, sw, &tot);
        run += tot;
        if (p < B) {
            vec_off[p] = off;
            dst_base[p] = off;
            dst_cap[p] = n;
            for (uint64_t i = off + n; i < off + len; i++) {
                keys[i] = 0xffffffffu;
                vals[i] = 0.0f;
            }
        }
    }
    if (threadIdx.x == 0) vec_off[B] = run;
}

cudaError_t last_status(uint32_t *d_status, cudaStream_t st, uint32_t *out) {
    PHYLO_CHECK(cudaMemcpyAsync(out, d_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    PHYLO_CHECK(cudaStreamSynchronize(st));
    return cudaSuccess;
}

}  // namespace

extern "C" {

// ---------------------------------------------------------------------------
// drop-in boundary
// ---------------------------------------------------------------------------

long estimateScratchMemory(const char *alphabet, int k, int max_vector_size) {
    // like the reference, any alphabet other than "DNA" is sized as protein
    const int alpha = (alphabet && strcmp(alphabet, "DNA") == 0) ? ALPHA_DNA : ALPHA_PROTEIN;
    const uint64_t max_size = max_vector_size > 0 ? (uint64_t)max_vector_size : 0;
    size_t need = compare_scratch_bytes(2 * max_size);
    BuildGeometry g;
    if (build_geometry(alpha, k, &g) == 0) {
        size_t b = build_scratch_bytes(g, 1, single_cand_cap(g, max_size));
        if (b > need) need = b;
    }
    return (long)need;
}

int buildCompositionVector(uintptr_t stream, uintptr_t d_temp_storage_ptr, long temp_storage_size,
                           const char *alphabet, int k, uintptr_t d_string_ptr, long string_len,
                           uintptr_t d_set_keys_ptr, uintptr_t d_set_values_ptr,
                           uintptr_t set_size_ptr, int max_vector_size) {
    const int alpha = parse_alphabet(alphabet);
    if (alpha < 0) {
        fprintf(stderr, "error: invalid alphabet '%s'\n", alphabet ? alphabet : "(null)");
        return (int)cudaErrorUnknown;
    }
    BuildGeometry g;
    const int gr = build_geometry(alpha, k, &g);
    if (gr == -1) {
        fprintf(stderr, "error: k=%d should be in range 3-10\n", k);
        return (int)cudaErrorUnknown;
    }
    if (gr == -2) {
        fprintf(stderr, "error: k=%d is too large for 32-bit keys with alphabet '%s'\n", k,
                alphabet);
        return (int)cudaErrorUnknown;
    }
    if (string_len < 0 || (uint64_t)string_len > 0xffffffffull || max_vector_size < 0 ||
        temp_storage_size < 0) {
        fprintf(stderr,
                "error: invalid sizes (string_len=%ld, max_vector_size=%d, "
                "temp_storage_size=%ld)\n",
                string_len, max_vector_size, temp_storage_size);
        return (int)cudaErrorInvalidValue;
    }
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t *h_size = (uint32_t *)set_size_ptr;
    const uint64_t max_size = (uint64_t)max_vector_size;
    BuildArgs a;
    memset(&a, 0, sizeof(a));
    cudaError_t err = build_carve(g, 1, single_cand_cap(g, max_size), (void *)d_temp_storage_ptr,
                                  (size_t)temp_storage_size, &a);
    if (err != cudaSuccess) {
        fprintf(stderr, "error: scratch of %ld bytes is smaller than the %zu bytes needed\n",
                temp_storage_size, build_scratch_bytes(g, 1, single_cand_cap(g, max_size)));
        return (int)err;
    }
    a.seq = (const uint8_t *)d_string_ptr;
    a.seq_off = a.seq_off_store;
    a.out_keys = (uint32_t *)d_set_keys_ptr;
    a.out_vals = (float *)d_set_values_ptr;
    a.single = 1;
    a.single_len = (uint64_t)string_len;
    a.single_cap = max_size;
    // the whole call's results: nnz, norm, candidates and status, in the order they have
    // in scratch; k_norm leaves them here where the device can write host memory
    SingleResult res = {};
    const bool direct = device_uses_host_memory();
    a.host_result = direct ? &res : nullptr;
    err = build_plan(a, st);
    if (err == cudaSuccess) err = build_emit(a, st);  // writes nothing where the checks below fail
    if (err != cudaSuccess) {
        cudaStreamSynchronize(st);  // what was queued may still write to res
        return (int)err;
    }
    if (!direct)
        PHYLO_CHECK(cudaMemcpyAsync(&res, a.nnz, sizeof(res), cudaMemcpyDeviceToHost, st));
    PHYLO_CHECK(cudaStreamSynchronize(st));
    if (h_size) *h_size = (uint32_t)res.nnz;
    if (res.status & DEV_CAPACITY) {
        fprintf(stderr,
                "error: candidate slots exceed the scratch capacity (%llu) for max_vector_size "
                "%d\n",
                (unsigned long long)a.cand_cap, max_vector_size);
        return (int)cudaErrorUnknown;
    }
    if (res.nnz > max_size) {
        fprintf(stderr,
                "error: size of composition vector (size: %llu) exceeds the given maximum (size: "
                "%d)\n",
                (unsigned long long)res.nnz, max_vector_size);
        return (int)cudaErrorUnknown;
    }
    return (int)cudaGetLastError();
}

// A pair compare and its status: `launch` queues the kernels, with the address they
// leave the status in (a host variable where the device can write it, else null).
}  // extern "C"

template <typename Launch>
static int compare_and_wait(cudaStream_t st, Launch launch) {
    uint32_t *d_status = nullptr;
    uint32_t status = DEV_WAIT_TIMEOUT;
    const bool direct = device_uses_host_memory();
    const cudaError_t e = launch(&d_status, direct ? &status : nullptr);
    if (e != cudaSuccess) {
        if (direct) cudaStreamSynchronize(st);  // what was queued may still write to status
        return (int)e;
    }
    if (direct) PHYLO_CHECK(cudaStreamSynchronize(st));
    else PHYLO_CHECK(last_status(d_status, st, &status));
    if (status) {
        fprintf(stderr, "error: compare kernel reported device status %u\n", status);
        return (int)cudaErrorLaunchTimeout;
    }
    return (int)cudaGetLastError();
}

extern "C" {

int compareCompositionVectors(uintptr_t stream, uintptr_t d_temp_storage_ptr, long temp_storage_size,
                              uintptr_t d_left_keys_ptr, uintptr_t d_left_values_ptr, int left_size,
                              uintptr_t d_right_keys_ptr, uintptr_t d_right_values_ptr,
                              int right_size, uintptr_t d_output_ptr) {
    if (left_size < 0 || right_size < 0 || temp_storage_size < 0) {
        fprintf(stderr, "error: negative size (vectors %d, %d; scratch %ld)\n", left_size,
                right_size, temp_storage_size);
        return (int)cudaErrorInvalidValue;
    }
    cudaStream_t st = (cudaStream_t)stream;
    return compare_and_wait(st, [&](uint32_t **d_status, uint32_t *host_status) -> cudaError_t {
        PHYLO_CHECK(compare_launch(st, (void *)d_temp_storage_ptr, (size_t)temp_storage_size,
                                   (const uint32_t *)d_left_keys_ptr,
                                   (const float *)d_left_values_ptr, (uint32_t)left_size,
                                   (const uint32_t *)d_right_keys_ptr,
                                   (const float *)d_right_values_ptr, (uint32_t)right_size,
                                   (double *)d_output_ptr, d_status, host_status));
        return cudaSuccess;
    });
}

// For callers that cannot allocate device memory (see include/phylogenetics.h):
// compareCompositionVectors on the library's built-in scratch array.
// Synchronous, like compareCompositionVectors.  No allocation of any kind.
int compareCompositionVectorsStatic(uintptr_t stream, uintptr_t d_left_keys_ptr,
                                    uintptr_t d_left_values_ptr, int left_size,
                                    uintptr_t d_right_keys_ptr, uintptr_t d_right_values_ptr,
                                    int right_size, uintptr_t d_output_ptr) {
    if (left_size < 0 || right_size < 0) {
        fprintf(stderr, "error: negative vector size (%d, %d)\n", left_size, right_size);
        return (int)cudaErrorInvalidValue;
    }
    cudaStream_t st = (cudaStream_t)stream;
    return compare_and_wait(st, [&](uint32_t **d_status, uint32_t *host_status) {
        return compare_launch_static(st, (const uint32_t *)d_left_keys_ptr,
                                     (const float *)d_left_values_ptr, (uint32_t)left_size,
                                     (const uint32_t *)d_right_keys_ptr,
                                     (const float *)d_right_values_ptr, (uint32_t)right_size,
                                     (double *)d_output_ptr, d_status, host_status);
    });
}

int phyloCompareTileElements(void) { return (int)compare_tile_elements(); }

// Test hook of the bounded waits (see include/phylogenetics.h).
void phyloCompareTestWaitLimit(unsigned int limit) { compare_set_first_wait_limit(limit); }

// ---------------------------------------------------------------------------
// batched construction (new)
// ---------------------------------------------------------------------------

// Scratch for building up to max_proteomes proteomes whose candidate slots sum
// to at most max_candidates.
long phyloBuildBatchScratch(const char *alphabet, int k, int max_proteomes, long max_candidates) {
    const int alpha = parse_alphabet(alphabet);
    BuildGeometry g;
    if (alpha < 0 || build_geometry(alpha, k, &g) != 0 || max_proteomes <= 0 || max_candidates < 0)
        return -1;
    return (long)build_scratch_bytes(g, max_proteomes, (uint64_t)max_candidates);
}

// Phase 1: counts, candidate slots, alpha, norms and per-proteome sizes.
// d_seq: concatenated sequence bytes; d_seq_off: uint64[num_proteomes + 1].
// h_nnz (host, num_proteomes entries) receives the vector sizes; h_candidates
// (host, may be null) the total candidate slots.  Synchronous.
int phyloBuildBatchPlan(uintptr_t stream, uintptr_t d_scratch, long scratch_size,
                        const char *alphabet, int k, int num_proteomes, uintptr_t d_seq,
                        uintptr_t d_seq_off, long max_candidates, int64_t *h_nnz,
                        int64_t *h_candidates) {
    const int alpha = parse_alphabet(alphabet);
    BuildGeometry g;
    if (alpha < 0 || build_geometry(alpha, k, &g) != 0 || num_proteomes <= 0 ||
        max_candidates < 0 || scratch_size < 0) {
        fprintf(stderr, "error: invalid batch build arguments (alphabet %s, k=%d, n=%d)\n",
                alphabet ? alphabet : "(null)", k, num_proteomes);
        return (int)cudaErrorInvalidValue;
    }
    cudaStream_t st = (cudaStream_t)stream;
    BuildArgs a;
    memset(&a, 0, sizeof(a));
    PHYLO_CHECK(build_carve(g, num_proteomes, (uint64_t)max_candidates, (void *)d_scratch,
                            (size_t)scratch_size, &a));
    a.seq = (const uint8_t *)d_seq;
    a.seq_off = (const uint64_t *)d_seq_off;
    PHYLO_CHECK(build_plan(a, st));
    PHYLO_CHECK(cudaMemcpyAsync(h_nnz, a.nnz, sizeof(uint64_t) * num_proteomes,
                                cudaMemcpyDeviceToHost, st));
    if (h_candidates)
        PHYLO_CHECK(cudaMemcpyAsync(h_candidates, a.cand_total, sizeof(uint64_t),
                                    cudaMemcpyDeviceToHost, st));
    uint32_t status = 0;
    PHYLO_CHECK(last_status(a.status, st, &status));
    if (status & DEV_CAPACITY) {
        fprintf(stderr, "error: candidate slots exceed max_candidates=%ld\n", max_candidates);
        return (int)cudaErrorMemoryAllocation;
    }
    return (int)cudaGetLastError();
}

// Phase 1 without waiting: the same kernels, then copies of the results into
// the caller's pinned host buffer h_summary (see the header); the caller
// synchronises the stream (or an event recorded after this call) before
// reading it.
int phyloBuildBatchPlanAsync(uintptr_t stream, uintptr_t d_scratch, long scratch_size,
                             const char *alphabet, int k, int num_proteomes, uintptr_t d_seq,
                             uintptr_t d_seq_off, long max_candidates, void *h_summary) {
    const int alpha = parse_alphabet(alphabet);
    BuildGeometry g;
    if (alpha < 0 || build_geometry(alpha, k, &g) != 0 || num_proteomes <= 0 || !h_summary ||
        max_candidates < 0 || scratch_size < 0) {
        fprintf(stderr, "error: invalid batch build arguments (alphabet %s, k=%d, n=%d)\n",
                alphabet ? alphabet : "(null)", k, num_proteomes);
        return (int)cudaErrorInvalidValue;
    }
    cudaStream_t st = (cudaStream_t)stream;
    BuildArgs a;
    memset(&a, 0, sizeof(a));
    PHYLO_CHECK(build_carve(g, num_proteomes, (uint64_t)max_candidates, (void *)d_scratch,
                            (size_t)scratch_size, &a));
    a.seq = (const uint8_t *)d_seq;
    a.seq_off = (const uint64_t *)d_seq_off;
    PHYLO_CHECK(build_plan(a, st));
    // summary layout, in scratch as in the caller's buffer: int64 nnz[B] | float64 norm[B] |
    // int64 candidates | uint32 status
    PHYLO_CHECK(cudaMemcpyAsync(h_summary, a.nnz, 16 * (size_t)num_proteomes + 12,
                                cudaMemcpyDeviceToHost, st));
    return (int)cudaGetLastError();
}

long phyloBuildBatchSummaryBytes(int num_proteomes) {
    return num_proteomes > 0 ? 16L * num_proteomes + 16 : -1;
}

// Phase 2 (after Plan, same scratch): writes vector p at
// d_keys/d_values[vec_off[p] ..], vec_off[p] = arena_base + sum of earlier sizes
// rounded up to 4 entries; d_vec_off (uint64[num_proteomes + 1]) receives the
// offsets.  Padding entries get key 0xffffffff and value 0.  Asynchronous.
int phyloBuildBatchEmit(uintptr_t stream, uintptr_t d_scratch, long scratch_size,
                        const char *alphabet, int k, int num_proteomes, long max_candidates,
                        uintptr_t d_keys, uintptr_t d_values, uintptr_t d_vec_off,
                        long arena_base, uintptr_t d_union_bits) {
    const int alpha = parse_alphabet(alphabet);
    BuildGeometry g;
    if (alpha < 0 || build_geometry(alpha, k, &g) != 0 || num_proteomes <= 0 ||
        max_candidates < 0 || scratch_size < 0 || arena_base < 0)
        return (int)cudaErrorInvalidValue;
    cudaStream_t st = (cudaStream_t)stream;
    BuildArgs a;
    memset(&a, 0, sizeof(a));
    PHYLO_CHECK(build_carve(g, num_proteomes, (uint64_t)max_candidates, (void *)d_scratch,
                            (size_t)scratch_size, &a));
    a.out_keys = (uint32_t *)d_keys;
    a.out_vals = (float *)d_values;
    a.union_bits = (uint32_t *)d_union_bits;
    uint64_t *vec_off = (uint64_t *)d_vec_off;
    k_arena_offsets<<<1, AO_THREADS, 0, st>>>(a.nnz, num_proteomes, (uint64_t)arena_base, vec_off,
                                              a.dst_base, a.dst_cap, a.out_keys, a.out_vals);
    PHYLO_CHECK(cudaGetLastError());
    PHYLO_CHECK(build_emit(a, st));
    return (int)cudaGetLastError();
}

// Per-proteome norms (sum of alpha^2) of the last Plan, double[num_proteomes].
int phyloBuildBatchNorms(uintptr_t stream, uintptr_t d_scratch, long scratch_size,
                         const char *alphabet, int k, int num_proteomes, long max_candidates,
                         double *h_norms) {
    const int alpha = parse_alphabet(alphabet);
    BuildGeometry g;
    if (alpha < 0 || build_geometry(alpha, k, &g) != 0 || num_proteomes <= 0 ||
        max_candidates < 0 || scratch_size < 0 || !h_norms)
        return (int)cudaErrorInvalidValue;
    BuildArgs a;
    memset(&a, 0, sizeof(a));
    PHYLO_CHECK(build_carve(g, num_proteomes, (uint64_t)max_candidates, (void *)d_scratch,
                            (size_t)scratch_size, &a));
    cudaStream_t st = (cudaStream_t)stream;
    PHYLO_CHECK(cudaMemcpyAsync(h_norms, a.norm, sizeof(double) * num_proteomes,
                                cudaMemcpyDeviceToHost, st));
    PHYLO_CHECK(cudaStreamSynchronize(st));
    return 0;
}

// Dense (K-1)- and (K-2)-mer count tables and n0/n1/n2 of proteome p of the last
// Plan (for count-parity checks).  Synchronous.
// Compact count table of proteome p (entry pw[w].x + rank of the bit in word w for
// every set bit of the seen bitmap's nw words; its count is the first of its `stride`
// words) expanded into a dense host table of `len` entries.
static cudaError_t expand_compact_counts(const uint32_t *d_seen, const uint2 *d_pw,
                                         const uint32_t *d_counts, int stride, uint64_t cap,
                                         uint64_t nw,
                                         int p, uint64_t len, uint32_t *h_out, cudaStream_t st) {
    std::vector<uint32_t> seen(nw);
    std::vector<uint2> pw(nw);
    PHYLO_CHECK(cudaMemcpyAsync(seen.data(), d_seen + (uint64_t)p * nw, sizeof(uint32_t) * nw,
                                cudaMemcpyDeviceToHost, st));
    PHYLO_CHECK(cudaMemcpyAsync(pw.data(), d_pw + (uint64_t)p * nw, sizeof(uint2) * nw,
                                cudaMemcpyDeviceToHost, st));
    PHYLO_CHECK(cudaStreamSynchronize(st));
    // ranks are kept for the words that hold seen bits
    uint64_t first = 0, n = 0;
    for (uint64_t w = 0; w < nw; w++) {
        if (n == 0 && seen[w]) first = pw[w].x;
        n += (uint64_t)__builtin_popcount(seen[w]);
    }
    if (first + n > cap) return cudaErrorInvalidValue;  // the build ran out of room
    std::vector<uint32_t> cc(n ? n * stride : 1);
    if (n)
        PHYLO_CHECK(cudaMemcpyAsync(cc.data(), d_counts + first * stride, sizeof(uint32_t) * n * stride,
                                    cudaMemcpyDeviceToHost, st));
    PHYLO_CHECK(cudaStreamSynchronize(st));
    memset(h_out, 0, sizeof(uint32_t) * len);
    for (uint64_t w = 0; w < nw; w++) {
        uint32_t bits = seen[w], r = bits ? pw[w].x - (uint32_t)first : 0u;
        while (bits) {
            const int j = __builtin_ctz(bits);
            bits &= bits - 1;
            if (w * 32 + j < len) h_out[w * 32 + j] = cc[(size_t)r * stride];
            r++;
        }
    }
    return cudaSuccess;
}

int phyloBuildBatchCounts(uintptr_t stream, uintptr_t d_scratch, long scratch_size,
                          const char *alphabet, int k, int num_proteomes, long max_candidates,
                          int p, uint32_t *h_c1, uint32_t *h_c2, uint32_t *h_tot) {
    const int alpha = parse_alphabet(alphabet);
    BuildGeometry g;
    if (alpha < 0 || build_geometry(alpha, k, &g) != 0 || p < 0 || p >= num_proteomes ||
        max_candidates < 0 || scratch_size < 0 || !h_c1 || !h_c2 || !h_tot)
        return (int)cudaErrorInvalidValue;
    BuildArgs a;
    memset(&a, 0, sizeof(a));
    PHYLO_CHECK(build_carve(g, num_proteomes, (uint64_t)max_candidates, (void *)d_scratch,
                            (size_t)scratch_size, &a));
    cudaStream_t st = (cudaStream_t)stream;
    if (a.compact1) {
        PHYLO_CHECK(expand_compact_counts(a.seen1, a.pw1, (const uint32_t *)a.cc, 2, a.cap1, g.T1s / 32, p, g.T1, h_c1, st));
    } else {
        PHYLO_CHECK(cudaMemcpyAsync(h_c1, a.c1 + (uint64_t)p * g.T1s, sizeof(uint32_t) * g.T1,
                                    cudaMemcpyDeviceToHost, st));
    }
    if (a.compact2) {
        PHYLO_CHECK(expand_compact_counts(a.seen2, a.pw2, a.c2, 1, a.cap2, g.T2s / 32, p, g.T2, h_c2, st));
    } else {
        PHYLO_CHECK(cudaMemcpyAsync(h_c2, a.c2 + (uint64_t)p * g.T2, sizeof(uint32_t) * g.T2,
                                    cudaMemcpyDeviceToHost, st));
    }
    PHYLO_CHECK(cudaMemcpyAsync(h_tot, a.tot + (uint64_t)p * 4, sizeof(uint32_t) * 3,
                                cudaMemcpyDeviceToHost, st));
    PHYLO_CHECK(cudaStreamSynchronize(st));
    return 0;
}

int phyloBuildLaunchesPerBatch(void) { return build_launches_per_batch(); }

// ---------------------------------------------------------------------------
// pair engine (new)
// ---------------------------------------------------------------------------

// Window index of an arena: roff uint32[num_vectors][R + 1], R = ceil(key_limit / 2^shift).
int phyloWindowIndex(uintptr_t stream, uintptr_t d_keys, uintptr_t d_vec_off, int num_vectors,
                     int window_shift, unsigned int num_windows, long max_vector_len,
                     uintptr_t d_roff) {
    if (num_vectors < 0 || window_shift < 0 || window_shift > 31 || max_vector_len < 0)
        return (int)cudaErrorInvalidValue;
    return (int)range_index_launch((const uint32_t *)d_keys, (const uint64_t *)d_vec_off,
                                   (uint32_t)num_vectors, num_windows, (uint32_t)window_shift,
                                   (uint32_t *)d_roff, (cudaStream_t)stream,
                                   (uint64_t)max_vector_len);
}

// Sets the kernel's shared-memory limit for this window width and reports the
// resident CTAs per SM.
int phyloPairsPrepare(int window_shift, int tile_rows, int tile_cols, int *ctas_per_sm) {
    if (!ap_shape_ok(tile_rows, tile_cols) || window_shift < 4 ||
        window_shift > ap_max_wshift(tile_rows, tile_cols))
        return (int)cudaErrorInvalidValue;
    return (int)ap_prepare((uint32_t)window_shift, tile_rows, tile_cols, ctas_per_sm);
}

int phyloPairsSmemBytes(int window_shift, int tile_rows, int tile_cols) {
    if (!ap_shape_ok(tile_rows, tile_cols)) return -1;
    return (int)ap_smem_bytes((uint32_t)window_shift, tile_rows, tile_cols);
}

int phyloPairsThreads(int window_shift, int tile_rows, int tile_cols) {
    if (!ap_shape_ok(tile_rows, tile_cols)) return -1;
    return ap_threads((uint32_t)window_shift, tile_rows, tile_cols);
}

// Launches the pair kernel over `num_items` items (8 uint32 each, see ApItem);
// row vectors come from the row arena, column vectors from the column arena
// (the same arena for all pairs of one set).  d_counter must be zero.
// d_item_cycles may be 0.
static int pairs_launch(uintptr_t stream, uintptr_t d_row_keys, uintptr_t d_row_values,
                        uintptr_t d_row_vec_off, uintptr_t d_row_roff, uintptr_t d_col_keys,
                        uintptr_t d_col_values, uintptr_t d_col_vec_off, uintptr_t d_col_roff,
                        unsigned int num_windows, int window_shift, uintptr_t d_rowids,
                        uintptr_t d_colids, uintptr_t d_items, int num_items, uintptr_t d_counter,
                        uintptr_t d_part, int fold, uintptr_t d_item_cycles, int tile_rows,
                        int tile_cols, int grid, bool parts) {
    // parts of at most eight or four rows are parts of 16-row tiles
    const int shape = parts && (tile_rows == 8 || tile_rows == 4) ? AP_TI : tile_rows;
    if (!ap_shape_ok(shape, tile_cols) || window_shift < 4 ||
        window_shift > ap_max_wshift(shape, tile_cols) || num_items < 0 || grid <= 0 ||
        (parts && (shape != AP_TI || tile_cols < 128)))
        return (int)cudaErrorInvalidValue;
    ApArgs a;
    a.row.keys = (const uint32_t *)d_row_keys;
    a.row.vals = (const float *)d_row_values;
    a.row.vec_off = (const uint64_t *)d_row_vec_off;
    a.row.roff = (const uint32_t *)d_row_roff;
    a.col.keys = (const uint32_t *)d_col_keys;
    a.col.vals = (const float *)d_col_values;
    a.col.vec_off = (const uint64_t *)d_col_vec_off;
    a.col.roff = (const uint32_t *)d_col_roff;
    a.R = num_windows;
    a.wshift = (uint32_t)window_shift;
    a.rowids = (const uint32_t *)d_rowids;
    a.colids = (const uint32_t *)d_colids;
    a.items = parts ? nullptr : (const ApItem *)d_items;
    a.subs = parts ? (const ApSubItem *)d_items : nullptr;
    a.nitems = (uint32_t)num_items;
    a.counter = (uint32_t *)d_counter;
    a.part = (FF *)d_part;
    // the 16-row kernel adds four products per accumulator between checks
    a.fold = fold >= 4 ? (uint32_t)fold & ~3u : (fold > 0 ? 4u : 28u);
    a.item_cycles = (int64_t *)d_item_cycles;
    return (int)ap_launch(a, tile_rows, tile_cols, grid, (cudaStream_t)stream);
}

int phyloPairsLaunch(uintptr_t stream, uintptr_t d_row_keys, uintptr_t d_row_values,
                     uintptr_t d_row_vec_off, uintptr_t d_row_roff, uintptr_t d_col_keys,
                     uintptr_t d_col_values, uintptr_t d_col_vec_off, uintptr_t d_col_roff,
                     unsigned int num_windows, int window_shift, uintptr_t d_rowids,
                     uintptr_t d_colids, uintptr_t d_items, int num_items, uintptr_t d_counter,
                     uintptr_t d_part, int fold, uintptr_t d_item_cycles, int tile_rows,
                     int tile_cols, int grid) {
    return pairs_launch(stream, d_row_keys, d_row_values, d_row_vec_off, d_row_roff, d_col_keys,
                        d_col_values, d_col_vec_off, d_col_roff, num_windows, window_shift,
                        d_rowids, d_colids, d_items, num_items, d_counter, d_part, fold,
                        d_item_cycles, tile_rows, tile_cols, grid, false);
}

// The same over parts of segments (12 uint32 each, see ApSubItem).
int phyloPairsLaunchParts(uintptr_t stream, uintptr_t d_row_keys, uintptr_t d_row_values,
                          uintptr_t d_row_vec_off, uintptr_t d_row_roff, uintptr_t d_col_keys,
                          uintptr_t d_col_values, uintptr_t d_col_vec_off, uintptr_t d_col_roff,
                          unsigned int num_windows, int window_shift, uintptr_t d_rowids,
                          uintptr_t d_colids, uintptr_t d_items, int num_items, uintptr_t d_counter,
                          uintptr_t d_part, int fold, uintptr_t d_item_cycles, int tile_rows,
                          int tile_cols, int grid) {
    return pairs_launch(stream, d_row_keys, d_row_values, d_row_vec_off, d_row_roff, d_col_keys,
                        d_col_values, d_col_vec_off, d_col_roff, num_windows, window_shift,
                        d_rowids, d_colids, d_items, num_items, d_counter, d_part, fold,
                        d_item_cycles, tile_rows, tile_cols, grid, true);
}

static int pairs_reduce(uintptr_t stream, uintptr_t d_part, uintptr_t d_tiles, int num_tiles,
                        int tile_words, int segments, int tile_rows, int tile_cols,
                        uintptr_t d_rowids, uintptr_t d_colids, uintptr_t d_out, long ldc,
                        int upper, int mirror) {
    if (!ap_shape_ok(tile_rows, tile_cols) || upper < 0 || upper > 2 || num_tiles < 0 ||
        (num_tiles > 0 && segments <= 0) || ldc <= 0)
        return (int)cudaErrorInvalidValue;
    ApReduceArgs r;
    r.part = (const FF *)d_part;
    r.tiles = (const uint32_t *)d_tiles;
    r.ntiles = (uint32_t)num_tiles;
    r.tile_words = (uint32_t)tile_words;
    r.S = (uint32_t)segments;
    r.ti = (uint32_t)tile_rows;
    r.tj = (uint32_t)tile_cols;
    r.rowids = (const uint32_t *)d_rowids;
    r.colids = (const uint32_t *)d_colids;
    r.out = (double *)d_out;
    r.ldc = (uint64_t)ldc;
    r.upper = upper;
    r.mirror = mirror;
    return (int)ap_reduce_launch(r, (cudaStream_t)stream);
}

// Sums the partial blocks of each tile (4 uint32 per tile: row0, nrow, col0, ncol).
int phyloPairsReduce(uintptr_t stream, uintptr_t d_part, uintptr_t d_tiles, int num_tiles,
                     int segments, int tile_rows, int tile_cols, uintptr_t d_rowids,
                     uintptr_t d_colids, uintptr_t d_out, long ldc, int upper, int mirror) {
    return pairs_reduce(stream, d_part, d_tiles, num_tiles, 4, segments, tile_rows, tile_cols,
                        d_rowids, d_colids, d_out, ldc, upper, mirror);
}

// The same for tiles with their own partial blocks (8 uint32 per tile: row0, nrow, col0,
// ncol, part0, nparts, two unused).
int phyloPairsReduceParts(uintptr_t stream, uintptr_t d_part, uintptr_t d_tiles, int num_tiles,
                          int tile_rows, int tile_cols, uintptr_t d_rowids, uintptr_t d_colids,
                          uintptr_t d_out, long ldc, int upper, int mirror) {
    return pairs_reduce(stream, d_part, d_tiles, num_tiles, 8, 1, tile_rows, tile_cols, d_rowids,
                        d_colids, d_out, ldc, upper, mirror);
}

// ---------------------------------------------------------------------------
// key-major (postings) pair engine (new)
// ---------------------------------------------------------------------------

long phyloPostingsSmemBytes(int block, int window_shift) {
    if (!pb_block_ok(block) || window_shift < 4 || window_shift > 14) return -1;
    const size_t n = pb_smem_bytes(block, (uint32_t)window_shift);
    return n ? (long)n : -1;
}

long phyloPostingsCapacity(int block, int window_shift) {
    if (!pb_block_ok(block) || window_shift < 4 || window_shift > 14) return -1;
    const uint32_t c = pb_capacity(block, (uint32_t)window_shift);
    return c ? (long)c : -1;
}

int phyloPostingsThreads(int block) { return pb_block_ok(block) ? pb_threads(block) : -1; }

int phyloPostingsPrepare(int block, int window_shift, int *ctas_per_sm) {
    if (phyloPostingsCapacity(block, window_shift) < 0) return (int)cudaErrorInvalidValue;
    return (int)pb_prepare(block, (uint32_t)window_shift, ctas_per_sm);
}

int phyloPostingsLaunch(uintptr_t stream, uintptr_t d_row_keys, uintptr_t d_row_values,
                        uintptr_t d_row_vec_off, uintptr_t d_row_roff, uintptr_t d_col_keys,
                        uintptr_t d_col_values, uintptr_t d_col_vec_off, uintptr_t d_col_roff,
                        unsigned int num_windows, int window_shift, uintptr_t d_rowids,
                        uintptr_t d_colids, uintptr_t d_items, int num_items, uintptr_t d_counter,
                        uintptr_t d_part, uintptr_t d_status, uintptr_t d_item_cycles, int block,
                        int grid) {
    if (phyloPostingsCapacity(block, window_shift) < 0 || num_items < 0 || grid <= 0)
        return (int)cudaErrorInvalidValue;
    if (num_items == 0) return 0;
    PbArgs a;
    a.row.keys = (const uint32_t *)d_row_keys;
    a.row.vals = (const float *)d_row_values;
    a.row.vec_off = (const uint64_t *)d_row_vec_off;
    a.row.roff = (const uint32_t *)d_row_roff;
    a.col.keys = (const uint32_t *)d_col_keys;
    a.col.vals = (const float *)d_col_values;
    a.col.vec_off = (const uint64_t *)d_col_vec_off;
    a.col.roff = (const uint32_t *)d_col_roff;
    a.R = num_windows;
    a.wshift = (uint32_t)window_shift;
    a.rowids = (const uint32_t *)d_rowids;
    a.colids = (const uint32_t *)d_colids;
    a.items = (const PbItem *)d_items;
    a.nitems = (uint32_t)num_items;
    a.counter = (uint32_t *)d_counter;
    a.part = (int64_t *)d_part;
    a.status = (uint32_t *)d_status;
    a.item_cycles = (int64_t *)d_item_cycles;
    return (int)pb_launch(a, block, grid, (cudaStream_t)stream);
}

int phyloPostingsReduce(uintptr_t stream, uintptr_t d_part, uintptr_t d_tiles, int num_tiles,
                        int block, uintptr_t d_rowids, uintptr_t d_colids, uintptr_t d_out,
                        long ldc, int self, int mirror) {
    if (!pb_block_ok(block) || num_tiles < 0 || ldc <= 0) return (int)cudaErrorInvalidValue;
    PbReduceArgs r;
    r.part = (const int64_t *)d_part;
    r.tiles = (const PbTile *)d_tiles;
    r.ntiles = (uint32_t)num_tiles;
    r.block = (uint32_t)block;
    r.rowids = (const uint32_t *)d_rowids;
    r.colids = (const uint32_t *)d_colids;
    r.out = (double *)d_out;
    r.ldc = (uint64_t)ldc;
    r.self = self;
    r.mirror = mirror;
    return (int)pb_reduce_launch(r, (cudaStream_t)stream);
}

long phyloKeyRankScratch(long key_limit) {
    if (key_limit <= 0 || key_limit > 0xffffffffl) return -1;
    return (long)rank_scratch_bytes((uint64_t)key_limit);
}

long phyloKeyRankBitmapBytes(long key_limit) {
    if (key_limit <= 0 || key_limit > 0xffffffffl) return -1;
    return (long)(rank_bitmap_words((uint64_t)key_limit) * sizeof(uint32_t));
}

int phyloKeyRanks(uintptr_t stream, uintptr_t d_scratch, long scratch_bytes, long key_limit,
                  uintptr_t d_keys, uintptr_t d_vec_off, int num_vectors, long max_vector_len,
                  uintptr_t d_union_bits, uintptr_t d_rank_keys, uintptr_t d_union_size) {
    if (key_limit <= 0 || key_limit > 0xffffffffl || num_vectors < 0 || max_vector_len < 0 ||
        scratch_bytes < (long)rank_scratch_bytes((uint64_t)key_limit))
        return (int)cudaErrorInvalidValue;
    return (int)key_ranks((const uint32_t *)d_keys, (const uint64_t *)d_vec_off,
                          (uint32_t)num_vectors, (uint64_t)max_vector_len, (uint64_t)key_limit,
                          (const uint32_t *)d_union_bits, (void *)d_scratch, (size_t)scratch_bytes,
                          (uint32_t *)d_rank_keys, (uint64_t *)d_union_size, (cudaStream_t)stream);
}

int phyloKeyRankIndex(uintptr_t stream, uintptr_t d_scratch, long scratch_bytes, long key_limit,
                      uintptr_t d_keys, uintptr_t d_vec_off, int num_vectors, long max_vector_len,
                      long arena_entries, uintptr_t d_union_bits, int window_shift,
                      unsigned int num_windows, uintptr_t d_rank_keys, uintptr_t d_roff) {
    if (key_limit <= 0 || key_limit > 0xffffffffl || num_vectors < 0 || window_shift < 0 ||
        window_shift > 31 || arena_entries < 0 || max_vector_len < 0 ||
        scratch_bytes < (long)rank_scratch_bytes((uint64_t)key_limit))
        return (int)cudaErrorInvalidValue;
    return (int)key_rank_index((const uint32_t *)d_keys, (const uint64_t *)d_vec_off,
                               (uint32_t)num_vectors, (uint64_t)max_vector_len,
                               (uint64_t)arena_entries, (uint64_t)key_limit,
                               (const uint32_t *)d_union_bits, (void *)d_scratch,
                               (size_t)scratch_bytes, (uint32_t)window_shift, num_windows,
                               (uint32_t *)d_rank_keys, (uint32_t *)d_roff, (cudaStream_t)stream);
}

int phyloSelfDot(uintptr_t stream, uintptr_t d_values, uintptr_t d_vec_off, int num_vectors,
                 long max_vector_len, uintptr_t d_part, uintptr_t d_out, long ldc) {
    if (num_vectors < 0 || max_vector_len < 0 || ldc <= 0) return (int)cudaErrorInvalidValue;
    return (int)self_dot_launch((const float *)d_values, (const uint64_t *)d_vec_off,
                                (uint32_t)num_vectors, (double *)d_out, (uint64_t)ldc,
                                (uint64_t)max_vector_len, (FF *)d_part, (cudaStream_t)stream);
}

long phyloSelfDotPartBytes(int num_vectors, long max_vector_len) {
    if (num_vectors < 0 || max_vector_len < 0) return -1;
    return (long)(self_dot_part_count((uint32_t)num_vectors, (uint64_t)max_vector_len) * sizeof(FF));
}

// Scratch bytes of phyloComparePairsMany for P pairs and at most max_tiles
// merge tiles (sum over pairs of ceil((nl + nr) / phyloCompareTileElements())).
long phyloComparePairsManyScratch(int num_pairs, long max_tiles) {
    if (num_pairs < 0 || max_tiles < 0) return -1;
    return (long)compare_many_scratch_bytes((uint32_t)num_pairs, (uint64_t)max_tiles);
}

// C of many pairs in one merge-path launch sequence: pair p compares vector
// pa[p] of the left arena with vector pb[p] of the right arena (arena =
// keys, values, uint64 offsets, uint32 sizes); results to d_out[p] (double).
// Asynchronous.
int phyloComparePairsMany(uintptr_t stream, uintptr_t d_scratch, long scratch_size,
                          uintptr_t d_lkeys, uintptr_t d_lvalues, uintptr_t d_loff,
                          uintptr_t d_lnnz, uintptr_t d_rkeys, uintptr_t d_rvalues,
                          uintptr_t d_roff, uintptr_t d_rnnz, uintptr_t d_pa, uintptr_t d_pb,
                          int num_pairs, long max_tiles, uintptr_t d_out) {
    if (num_pairs < 0 || max_tiles < 0 || scratch_size < 0) return (int)cudaErrorInvalidValue;
    return (int)compare_many_launch(
        (cudaStream_t)stream, (void *)d_scratch, (size_t)scratch_size, (const uint32_t *)d_lkeys,
        (const float *)d_lvalues, (const uint64_t *)d_loff, (const uint32_t *)d_lnnz,
        (const uint32_t *)d_rkeys, (const float *)d_rvalues, (const uint64_t *)d_roff,
        (const uint32_t *)d_rnnz, (const uint32_t *)d_pa, (const uint32_t *)d_pb,
        (uint32_t)num_pairs, (uint64_t)max_tiles, (double *)d_out, nullptr);
}

// Pair kernel launch on raw arena pointers for one pair, through the merge
// path, asynchronous (used by the batched engine for vectors whose values
// are not finite).  Scratch from estimateScratchMemory.
int phyloComparePairAsync(uintptr_t stream, uintptr_t d_scratch, long scratch_size,
                          uintptr_t d_left_keys, uintptr_t d_left_values, int left_size,
                          uintptr_t d_right_keys, uintptr_t d_right_values, int right_size,
                          uintptr_t d_out) {
    if (left_size < 0 || right_size < 0 || scratch_size < 0) return (int)cudaErrorInvalidValue;
    return (int)compare_launch((cudaStream_t)stream, (void *)d_scratch, (size_t)scratch_size,
                               (const uint32_t *)d_left_keys, (const float *)d_left_values,
                               (uint32_t)left_size, (const uint32_t *)d_right_keys,
                               (const float *)d_right_values, (uint32_t)right_size,
                               (double *)d_out, nullptr);
}

}  // extern "C"
