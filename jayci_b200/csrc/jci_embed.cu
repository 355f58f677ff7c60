// jci_embed.cu -- sigma of a truncated space through the full CI space of the
// same electrons and orbitals.
//
// With several occupation groups per spin the Hamiltonian of the space is the
// full space's Hamiltonian between the determinants that are kept, so
//   sigma = P H_full (c with zeros elsewhere),
// and the one-group plans (jci_fci.cu) compute H_full c: rows and columns of
// matrices, tensor-core products and coalesced reads, where the generic kernel
// (k_sigma_generic) walks both strings' excitation lists for every determinant
// and gathers single elements.  It pays while the full space is not too many
// times larger: measured per determinant, the generic kernel takes 5 to 17 ns
// and a full-space plan 0.4 to 0.8 ns, so up to kEmbedRatio = 16 the two are
// timed once per precision and space, and the faster one is kept.  The two sum
// in different orders; a caller that needs the same bits in every process
// reads the route and pins it (embed_route, embed_set_route).
// Measured: 12 electrons in 16 orbitals (2 DOCC, 10 active, 4 virtual,
// excitation level 2; 13.0 of 64.1 million determinants) FP64 215 -> 53.3 ms,
// FP32 188 -> 34.4; 11 electrons in 15 orbitals (2 DOCC, 9 active; 3.2 of 15.0
// million) FP64 40 -> 10.0 ms; 11 in 12 (1 DOCC, 7 active; 0.12 of 0.73
// million) 0.73 -> 0.48 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "jci_internal.h"
#include "jci_kernels.cuh"

namespace jci {

constexpr long long kEmbedRatio = 16;   // full over kept determinants, at most
constexpr int kEmbedStrings = 16384;    // full strings of a spin, at most
constexpr long long kEmbedMin = 16384;  // determinants: below, the generic kernel takes some 0.1 ms

struct Embedding {
    jci_space *full = nullptr;
    int *inv[2] = {nullptr, nullptr};   // [full string] string of the space, or -1
    void *v[2] = {nullptr, nullptr}, *o[2] = {nullptr, nullptr};  // full vectors, per precision
    int use[2] = {0, 0};                // per precision: 0 not timed, 1 this way, -1 the generic one
    bool none = false;                  // the space has no usable full space
    cudaEvent_t done = nullptr;         // the last sigma through the vectors and the full scratch
};

// The pair block, row and column of full element (ia, ib) as a position in the
// space's vector, or -1.
__device__ __forceinline__ long long embed_pos(const SpaceView &v, int p, int q) {
    if (p < 0 || q < 0) return -1;
    const int gp = v.a.grp[p], gq = v.b.grp[q];
    const int k = v.pairidx[gp * v.qegrps + gq];
    if (k < 0) return -1;
    return v.pqoff[k] + (long long)(p - v.a.gstart[gp]) * v.b.gnstr[gq] + (q - v.b.gstart[gq]);
}

// in: full = the space's vector with zeros elsewhere; out: the space's vector
// = the elements of full that it keeps.  One row of the full matrix per
// blockIdx.y; bound by the full matrix's one read or write.
template <typename T, bool IN>
__global__ void __launch_bounds__(256)
    k_embed(SpaceView v, const int *__restrict__ inva, const int *__restrict__ invb, int nb,
            T *__restrict__ full, T *__restrict__ vec) {
    if (v.skip && *v.skip) return;
    const int ib = blockIdx.x * 256 + threadIdx.x;
    if (ib >= nb) return;
    const int p = inva[blockIdx.y];
    T *f = full + (long long)blockIdx.y * nb + ib;
    const long long d = p < 0 ? -1 : embed_pos(v, p, invb[ib]);
    if (IN)
        *f = d < 0 ? T(0) : vec[d];
    else if (d >= 0)
        vec[d] = *f;
}

static void embed_drop(Embedding *e) {
    if (e->full) jci_space_destroy(e->full);
    e->full = nullptr;
    for (int k = 0; k < 2; k++) {
        cudaFree(e->inv[k]);
        cudaFree(e->v[k]);
        cudaFree(e->o[k]);
        e->inv[k] = nullptr;
        e->v[k] = e->o[k] = nullptr;
    }
}

void embed_free(DeviceState *d) {
    if (!d->emb) return;
    embed_drop(d->emb);
    if (d->emb->done) cudaEventDestroy(d->emb->done);
    delete d->emb;
    d->emb = nullptr;
}

int embed_generation(const DeviceState *d) {
    return d->emb && d->emb->full && d->emb->full->dev ? d->emb->full->dev->sigma_gen : 0;
}

jci_status embed_wait_status(const DeviceState *d) {
    return d->emb && d->emb->full ? fci_wait_status(d->emb->full) : JCI_OK;
}

static jci_status embed_integrals(jci_space *s) {
    Embedding *e = s->dev->emb;
    try {
        return jci_set_integrals(e->full, s->m1.data(), s->m2.data(), s->ci_orbs, s->nucrep,
                                 s->frzcore);
    } catch (const std::bad_alloc &) {
        return JCI_ERR_NOMEM;
    }
}

jci_status embed_set_integrals(jci_space *s) {
    Embedding *e = s->dev->emb;
    return e && e->full ? embed_integrals(s) : JCI_OK;
}

bool embed_strings(const jci_space *s, long long n[2]) {
    const int na = s->ci_aelec, nb = s->ci_belec, no = s->ci_orbs;
    if (s->ndets < kEmbedMin || no > 64 || na - nb < 0 || na - nb > 1) return false;
    n[0] = binom(no, na);
    n[1] = binom(no, nb);
    return n[0] >= 1 && n[1] >= 1 && n[0] <= kEmbedStrings && n[1] <= kEmbedStrings &&
           n[0] * n[1] <= kEmbedRatio * s->ndets;
}

// The full space and the string maps; false when there is none within the
// limits or the device's free memory.
static bool embed_try(jci_space *s) {
    DeviceState *d = s->dev;
    Embedding *e = d->emb;
    if (e->full) return true;
    const int na = s->ci_aelec, nb = s->ci_belec, no = s->ci_orbs;
    long long n[2];
    if (!embed_strings(s, n)) return false;
    const long long fa = n[0], fb = n[1];
    // vectors, transposes and digits of both precisions, and room to spare
    size_t mfree = 0, mtotal = 0;
    if (cudaMemGetInfo(&mfree, &mtotal) != cudaSuccess ||
        (size_t)fa * fb * 96 + (size_t(4) << 30) > mfree / 2) {
        cudaGetLastError();
        return false;
    }
    if (jci_space_create(na + nb, no, 0, 0, no, 0, 0, &e->full) != JCI_OK) {
        e->full = nullptr;
        return false;
    }
    bool ok = e->full->ci_aelec == na && e->full->ci_belec == nb && e->full->ci_orbs == no;
    for (int sp = 0; sp < 2 && ok; sp++) {
        const SpinSpace &x = s->sp[sp];
        std::vector<int> inv(e->full->sp[sp].nstr, -1);
        for (int i = 0; i < x.nstr && ok; i++) {
            const int f = string_index(e->full, sp, &x.istr[(size_t)i * x.nelec]);
            ok = f >= 0 && inv[f] < 0;
            if (ok) inv[f] = i;
        }
        ok = ok && cudaMalloc((void **)&e->inv[sp], inv.size() * sizeof(int)) == cudaSuccess &&
             cudaMemcpy(e->inv[sp], inv.data(), inv.size() * sizeof(int),
                        cudaMemcpyHostToDevice) == cudaSuccess;
    }
    ok = ok && embed_integrals(s) == JCI_OK && fci_supported(e->full);
    if (!ok) {
        cudaGetLastError();
        embed_drop(e);
        return false;
    }
    return true;
}

// Host memory that runs out is no usable full space either.
static bool embed_build(jci_space *s) {
    try {
        return embed_try(s);
    } catch (const std::bad_alloc &) {
        embed_drop(s->dev->emb);
        return false;
    }
}

// Every sigma of the handle goes through the one pair of full vectors and the
// full space's scratch, where the generic kernel has none: each waits for the
// one before it, on whatever stream that is.  In a capture the wait and the
// record become nodes of the graph.  The Davidson's captured iterations need
// neither: they follow an uncaptured sigma on the same stream, and the solve
// waits for them.
static jci_status embed_order(const DeviceState *d, Embedding *e, cudaStream_t st, bool after) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    JCI_CUDA(cudaStreamIsCapturing(st, &cs));
    const bool captured = cs != cudaStreamCaptureStatusNone;
    if (captured && st == d->stream) return JCI_OK;
    if (!e->done) JCI_CUDA(cudaEventCreateWithFlags(&e->done, cudaEventDisableTiming));
    if (after)
        JCI_CUDA(cudaEventRecordWithFlags(
            e->done, st, captured ? cudaEventRecordExternal : cudaEventRecordDefault));
    else
        JCI_CUDA(cudaStreamWaitEvent(st, e->done,
                                     captured ? cudaEventWaitExternal : cudaEventWaitDefault));
    return JCI_OK;
}

template <typename T>
static jci_status embed_run(jci_space *s, int nvec, const T *v, T *o, long long ld,
                            cudaStream_t st) {
    constexpr int prec = sizeof(T) == 8 ? 0 : 1;
    DeviceState *d = s->dev;
    Embedding *e = d->emb;
    const int fa = e->full->sp[0].nstr, fb = e->full->sp[1].nstr;
    SpaceView w = make_view(d);
    w.ndets = s->ndets;
    const dim3 g((fb + 255) / 256, fa);
    T *fv = (T *)e->v[prec], *fo = (T *)e->o[prec];
    e->full->dev->sigma_skip = d->sigma_skip;
    jci_status r = embed_order(d, e, st, false);
    if (r) return r;
    for (int k = 0; k < nvec; k++) {
        k_embed<T, true><<<g, 256, 0, st>>>(w, e->inv[0], e->inv[1], fb, fv,
                                            const_cast<T *>(v) + k * ld);
        r = fci_sigma(e->full, 1, fv, fo, (long long)fa * fb,
                                 prec == 0 ? JCI_FP64 : JCI_FP32, st);
        if (r) return r;
        k_embed<T, false><<<g, 256, 0, st>>>(w, e->inv[0], e->inv[1], fb, fo, o + k * ld);
    }
    JCI_CUDA(cudaGetLastError());
    return embed_order(d, e, st, true);
}

jci_status embed_sigma(jci_space *s, int nvec, const void *v, void *o, long long ld, int precision,
                       cudaStream_t st) {
    if (precision == JCI_FP32)
        return embed_run<float>(s, nvec, (const float *)v, (float *)o, ld, st);
    return embed_run<double>(s, nvec, (const double *)v, (double *)o, ld, st);
}

// Full-space vectors of one precision.
static bool embed_vectors(Embedding *e, int prec) {
    const size_t n = (size_t)e->full->sp[0].nstr * e->full->sp[1].nstr;
    const size_t w = prec ? sizeof(float) : sizeof(double);
    const bool ok = (e->v[prec] || cudaMalloc(&e->v[prec], n * w) == cudaSuccess) &&
                    (e->o[prec] || cudaMalloc(&e->o[prec], n * w) == cudaSuccess);
    if (!ok) cudaGetLastError();
    return ok;
}

// A precision that does not come through here lets go of its vectors, and of
// the full space unless the other one does (a later precision builds it again).
static void embed_unused(DeviceState *d, int prec) {
    Embedding *e = d->emb;
    d->sigma_gen++;
    cudaFree(e->v[prec]);
    cudaFree(e->o[prec]);
    e->v[prec] = e->o[prec] = nullptr;
    if (e->use[prec ^ 1] <= 0) embed_drop(e);
}

// Whether sigma of this space runs through the full space; on the first call
// of a precision (never while the stream is being captured) times one vector
// both ways, on the caller's buffers.
bool embed_chosen(jci_space *s, const void *v, void *o, long long ld, int precision,
                  cudaStream_t st) {
    DeviceState *d = s->dev;
    const int prec = precision == JCI_FP32 ? 1 : 0;
    if (!d->emb) d->emb = new (std::nothrow) Embedding();
    Embedding *e = d->emb;
    if (!e) return false;
    if (e->use[prec] || e->none) return e->use[prec] > 0;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
        return false;
    if (!embed_build(s)) {
        e->none = true;
        return false;
    }
    e->use[prec] = -1;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    bool ok = embed_vectors(e, prec) && cudaEventCreate(&e0) == cudaSuccess &&
              cudaEventCreate(&e1) == cudaSuccess;
    const int *skip = d->sigma_skip;
    d->sigma_skip = nullptr;
    auto best = [&](auto fn) {
        float m = 1e30f;
        for (int k = 0; ok && k < 3; k++) {
            if (k == 0) ok = fn() == JCI_OK;  // first use: tables, plans
            cudaEventRecord(e0, st);
            ok = ok && fn() == JCI_OK;
            cudaEventRecord(e1, st);
            float t = 1e30f;
            ok = ok && cudaEventSynchronize(e1) == cudaSuccess &&
                 cudaEventElapsedTime(&t, e0, e1) == cudaSuccess;
            m = std::min(m, t);
            if (t > 50.f) break;
        }
        return m;
    };
    const float full = best([&] { return embed_sigma(s, 1, v, o, ld, precision, st); });
    const bool full_ok = ok;
    ok = true;
    const float gen = full_ok ? best([&] { return device_sigma_generic(s, 1, v, o, ld, precision, st); })
                              : 0.f;
    d->sigma_skip = skip;
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaGetLastError();
    if (full_ok && ok && full < gen) {
        e->use[prec] = 1;
        return true;
    }
    embed_unused(d, prec);
    return false;
}

void embed_route(const DeviceState *d, int precision, int *route, int *mode, int *nt, int *R,
                 int *B) {
    const int prec = precision == JCI_FP32 ? 1 : 0;
    const Embedding *e = d ? d->emb : nullptr;
    float ms;
    *route = *mode = *nt = *R = *B = 0;
    if (!e) return;
    // without a usable full space there is only the generic kernel
    *route = e->use[prec] > 0 ? kRouteFull
             : e->use[prec] < 0 || e->none ? kRouteGeneric : kRouteTimed;
    if (*route == kRouteFull) fci_tuning(e->full, precision, mode, nt, R, B, &ms);
}

jci_status embed_set_route(jci_space *s, int precision, int route, int mode, int nt, int R, int B) {
    DeviceState *d = s->dev;
    const int prec = precision == JCI_FP32 ? 1 : 0;
    if (!d->emb) d->emb = new (std::nothrow) Embedding();
    Embedding *e = d->emb;
    if (!e) return JCI_ERR_NOMEM;
    // nothing that is let go of is still in use
    JCI_CUDA(cudaStreamSynchronize(d->stream));
    if (e->done) JCI_CUDA(cudaEventSynchronize(e->done));
    if (route == kRouteFull) {
        if (!embed_build(s)) return JCI_ERR_ARG;
        jci_status r = embed_vectors(e, prec) ? JCI_OK : JCI_ERR_NOMEM;
        // all 0: the full space's own autotuner
        if (!r && (mode || nt || R || B))
            r = fci_force_plan(e->full, precision, mode, nt, R, B);
        if (r) {
            if (e->use[prec] <= 0) embed_unused(d, prec);
            return r;
        }
        e->use[prec] = 1;
        d->sigma_gen++;
        return JCI_OK;
    }
    e->use[prec] = route == kRouteGeneric ? -1 : 0;
    embed_unused(d, prec);
    if (route == kRouteTimed) e->none = false;
    return JCI_OK;
}

}  // namespace jci
