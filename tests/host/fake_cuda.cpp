// A CUDA runtime without a device, for the library's host code: device memory
// is host memory of a bounded amount, kernels do nothing, and every launch is
// recorded with what it is ordered behind (vector clocks over the streams), so
// that a launch which may read an array before the launch that writes it has
// ended is counted (fake_races).  All streams but null count as non-blocking.
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <string>
#include <vector>

#include "ivr_handles.h"
#include "ivr_mlp.h"

namespace {

using Clock = std::map<int, int>;  // stream -> launches of it that have ended
void join(Clock &a, const Clock &b)
{
    for (auto &e : b) a[e.first] = std::max(a[e.first], e.second);
}

struct Stream {
    int id;
    Clock clock;       // what the stream's next launch is ordered behind
    Clock before;      // ... and what a launch that may begin before the last one has ended is
    bool capturing = false;
};
struct Event {
    Clock clock;
};
struct Op {
    int stream = -1, seq = 0;
};

struct State {
    std::vector<Stream *> streams;
    Stream legacy{0};
    int next_stream = 1;
    Clock host;                     // what the host has waited for
    std::map<const void *, Op> writer;
    std::map<const void *, std::vector<Op>> readers;  // since that write
    int races = 0;
    std::string first;              // the first of them
    std::map<void *, size_t> live;  // device allocations
    size_t in_use = 0, capacity = ~(size_t) 0;
    long mallocs = 0, fail_malloc = -1, fail_more = 0, fail_launch = -1, launches = 0, early = 0;
    cudaError_t last = cudaSuccess;
} g;

Stream &of(cudaStream_t s) { return s ? *(Stream *) s : g.legacy; }
cudaError_t error(cudaError_t e)
{
    if (e != cudaSuccess) g.last = e;
    return e;
}
void all_done()
{
    join(g.host, g.legacy.clock);
    for (auto *s : g.streams) join(g.host, s->clock);
}

bool covers(const Clock &c, const Op &o)
{
    auto it = c.find(o.stream);
    return it != c.end() && it->second >= o.seq;
}
void race(const char *what, const char *who)
{
    if (g.races++ == 0) g.first = std::string(who) + ": " + what;
}

// One launch, copy or memset on s, with what it reads and writes.
struct Launch {
    Stream &s;
    Clock sees;
    Op op;
    const char *who;
    Launch(cudaStream_t st, const char *name, bool early = false) : s(of(st)), who(name)
    {
        join(s.clock, g.host);
        sees = early ? s.before : s.clock;
        join(sees, g.host);
        s.before = s.clock;
        op.stream = s.id;
        op.seq = ++s.clock[s.id];
        g.early += early;
    }
    Launch &read(const void *p)
    {
        auto w = p ? g.writer.find(p) : g.writer.end();
        if (w != g.writer.end() && !covers(sees, w->second)) race("reads what may not be written yet", who);
        if (p) g.readers[p].push_back(op);
        return *this;
    }
    Launch &write(const void *p)
    {
        if (!p) return *this;
        auto w = g.writer.find(p);
        if (w != g.writer.end() && !covers(sees, w->second)) race("writes what may still be written", who);
        for (auto &r : g.readers[p])
            if (!covers(sees, r)) race("writes what may still be read", who);
        g.readers[p].clear();
        g.writer[p] = op;
        return *this;
    }
    // as the launchers do: what cudaGetLastError has to say
    cudaError_t done()
    {
        if (g.fail_launch >= 0 && g.fail_launch-- == 0) error(cudaErrorLaunchOutOfResources);
        g.launches++;
        return cudaGetLastError();
    }
};
// a memset or copy: no kernel, so no launch behind it begins early
void full(cudaStream_t st)
{
    Stream &s = of(st);
    s.before = s.clock;
}

}  // namespace

extern "C" {

void fake_reset(void)
{
    g.races = 0;
    g.first.clear();
    g.writer.clear();
    g.readers.clear();
    g.mallocs = g.launches = g.early = 0;
    g.fail_malloc = g.fail_launch = -1;
    g.fail_more = 0;
    g.capacity = ~(size_t) 0;
    g.last = cudaSuccess;
}
int fake_races(void) { return g.races; }
const char *fake_first_race(void) { return g.first.c_str(); }
size_t fake_in_use(void) { return g.in_use; }
long fake_mallocs(void) { return g.mallocs; }
long fake_launches(void) { return g.launches; }
long fake_early(void) { return g.early; }
void fake_capacity(size_t n) { g.capacity = n; }
// the n-th allocation from now fails (0: the next one), and `more` behind it
void fake_fail_malloc(long n) { g.fail_malloc = n; }
void fake_fail_more(long n) { g.fail_more = n; }
void fake_fail_launch(long n) { g.fail_launch = n; }

cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = g.last;
    g.last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "an error"; }

cudaError_t cudaMalloc(void **p, size_t n)
{
    g.mallocs++;
    const bool fails = g.fail_malloc == 0;
    if (g.fail_malloc > 0 || (fails && g.fail_more-- == 0)) g.fail_malloc--;
    if (fails || n > g.capacity - std::min(g.capacity, g.in_use))
        return error(cudaErrorMemoryAllocation);
    if (posix_memalign(p, 512, (n + 511) / 512 * 512)) return error(cudaErrorMemoryAllocation);
    memset(*p, 0, n);
    g.live[*p] = n;
    g.in_use += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    if (!p) return cudaSuccess;
    all_done();
    auto it = g.live.find(p);
    if (it == g.live.end()) abort();  // not, or no longer, an allocation
    for (auto w = g.writer.lower_bound(p); w != g.writer.end() && (char *) w->first < (char *) p + it->second;)
        w = g.writer.erase(w);
    for (auto r = g.readers.lower_bound(p); r != g.readers.end() && (char *) r->first < (char *) p + it->second;)
        r = g.readers.erase(r);
    g.in_use -= it->second;
    g.live.erase(it);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *, const void *) { return cudaErrorInvalidValue; }

cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st)
{
    Launch(st, "copy").read(s).write(d);
    full(st);
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k)
{
    cudaMemcpyAsync(d, s, n, k, nullptr);
    join(g.host, g.legacy.clock);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st)
{
    Launch(st, "memset").write(d);
    full(st);
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    Stream *q = new Stream{g.next_stream++};
    g.streams.push_back(q);
    *s = (cudaStream_t) q;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long *id) { *id = (unsigned long long) of(s).id; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *st)
{
    *st = of(s).capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    join(g.host, of(s).clock);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void)
{
    all_done();
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    if (of(s).capturing) return error(cudaErrorStreamCaptureIsolation);  // an event from outside the capture
    join(of(s).clock, ((Event *) e)->clock);
    full(s);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t) new Event(); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Event *) e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    ((Event *) e)->clock = of(s).clock;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { join(g.host, ((Event *) e)->clock); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { of(s).capturing = true; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *gr)
{
    of(s).capturing = false;
    *gr = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) { *x = (cudaGraphExec_t) 1; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

cudaChannelFormatDesc cudaCreateChannelDesc(int x, int y, int z, int w, cudaChannelFormatKind f)
{
    return cudaChannelFormatDesc{x, y, z, w, f};
}
cudaError_t cudaMalloc3DArray(cudaArray_t *, const cudaChannelFormatDesc *, cudaExtent, unsigned) { return error(cudaErrorNotSupported); }
cudaError_t cudaMemcpy3D(const cudaMemcpy3DParms *) { return error(cudaErrorNotSupported); }
cudaError_t cudaFreeArray(cudaArray_t) { return cudaSuccess; }
cudaError_t cudaCreateTextureObject(cudaTextureObject_t *, const cudaResourceDesc *, const cudaTextureDesc *,
                                    const cudaResourceViewDesc *)
{
    return error(cudaErrorNotSupported);
}
cudaError_t cudaDestroyTextureObject(cudaTextureObject_t) { return cudaSuccess; }

}  // extern "C"

namespace ivr {

namespace {
long long tiles(const FrameDesc &f) { return (long long) ((f.out_w + 7) >> 3) * ((f.out_h + 3) >> 2); }
}  // namespace

size_t dtype_size(int dtype) { return dtype == IVR_F32 ? 4 : dtype == IVR_U16 ? 2 : 1; }
cudaError_t launch_byteswap(void *d, long long, int, cudaStream_t s) { return Launch(s, "byteswap").write(d).done(); }
cudaError_t launch_gather_brick(const void *src, int, int, int, void *d, int, int, int, int, int, int, int, cudaStream_t s)
{
    return Launch(s, "gather").read(src).write(d).done();
}
cudaError_t launch_minmax(const void *d, int, long long, float *p, int, cudaStream_t s)
{
    return Launch(s, "minmax").read(d).write(p).done();
}
cudaError_t launch_histogram(const void *d, int, long long, float, int, int *h, cudaStream_t s)
{
    return Launch(s, "histogram").read(d).write(h).done();
}
cudaError_t launch_macrocells(const void *d, int, int, int, int, int, float *mc, int, int, int, cudaStream_t s)
{
    return Launch(s, "macrocells").read(d).write(mc).done();
}
cudaError_t launch_empty_flags(const float *mc, int, int, int, const int *nz, const double *ap, int, int, float,
                               uint8_t *empty, uint8_t *opac, cudaStream_t s)
{
    return Launch(s, "empty flags").read(mc).read(nz).read(ap).write(empty).write(opac).done();
}
cudaError_t launch_dist_transform(uint8_t *d, int, int, int, cudaStream_t s) { return Launch(s, "distances").write(d).done(); }
cudaError_t launch_gradient(const void *d, int, int, int, int, float4 *o, cudaStream_t s)
{
    return Launch(s, "gradient").read(d).write(o).done();
}
size_t quad_bytes(int dtype, int nx, int ny, int nz) { return (size_t) (nx - 1) * (ny - 1) * nz * 4 * dtype_size(dtype); }
cudaError_t launch_quads(const void *d, int, int, int, int, void *q, cudaStream_t s)
{
    return Launch(s, "quads").read(d).write(q).done();
}
cudaError_t launch_composite(float *d, const float *src, int, long long, cudaStream_t s)
{
    return Launch(s, "composite").read(src).write(d).done();
}
cudaError_t launch_quantize(const float *in, uint8_t *out, long long, cudaStream_t s)
{
    return Launch(s, "quantize").read(in).write(out).done();
}
int minmax_parts() { return 8; }
cudaError_t noalloc_histogram(const void *, int, long long, int, int *, float *, cudaStream_t) { return error(cudaErrorNotSupported); }

bool tile_order_pays(const FrameDesc &f) { return tiles(f) >= 24320; }
long long judge_scratch_bytes(const FrameDesc &f)
{
    const long long n = tiles(f);
    return n > f.judge_phase ? (n - f.judge_phase + f.judge_stride - 1) / f.judge_stride * 128 : 0;
}
cudaError_t launch_march(const FrameDesc &f, float4 *, uchar4 *, cudaStream_t s, long long *tickets, bool early)
{
    if (tickets) *tickets = tiles(f);
    Launch l(s, f.judge ? "judged march" : f.gate ? "gated march" : f.census ? "census march" : "plain march", early);
    l.read(f.lut).read(f.perm).read(f.learned_bad);
    for (int k = 0; k < f.nb; k++) {
        l.read(f.b[k].data).read(f.b[k].quad).read(f.b[k].empty);
        if (f.judge) l.read(f.exact[k]);
    }
    return l.done();
}
cudaError_t launch_judge_compare(const FrameDesc &, const uchar4 *, const float4 *, cudaStream_t s)
{
    return Launch(s, "judge compare").done();
}
cudaError_t launch_tile_order(const FrameDesc &f, uint8_t *key, int *counts, int *perm, cudaStream_t s)
{
    Launch l(s, "tile order");
    for (int k = 0; k < f.nb; k++) l.read(f.b[k].empty).read(f.b[k].opac);
    return l.write(key).write(counts).write(perm).done();
}
cudaError_t launch_batch(int, int, const BatchHeader *hdr, const BatchItem *items, unsigned long long *, cudaStream_t s)
{
    Launch l(s, "batch");
    l.read(hdr);
    for (int i = 0; i < hdr->nitems; i++)
        for (int k = 0; k < items[i].f.nb; k++) l.read(items[i].f.b[k].empty);
    return l.done();
}
int batch_variant_tile_w(int) { return 8; }
cudaError_t launch_sample_peak(const FrameDesc &, int, const SamplerTex &, int, float4 *, long long *, unsigned *, cudaStream_t)
{
    return error(cudaErrorNotSupported);
}
int sample_peak_threads() { return 32; }

cudaError_t mlp_forward(const MlpDev &, const void *x, long long, float *y, cudaStream_t s)
{
    return Launch(s, "forward").read(x).write(y).done();
}
cudaError_t mlp_train_step(const MlpDev &, const void *x, const float *t, const int *idx, long long, long long, float,
                           float, float *grad, float *, cudaStream_t s)
{
    return Launch(s, "train step").read(x).read(t).read(idx).write(grad).done();
}
cudaError_t mlp_adam(float *p, float *, float *, float *grad, float, int, const float *c12, void *, void *, void *,
                     cudaStream_t s)
{
    return Launch(s, "adam").read(c12).write(grad).write(p).done();
}
void mlp_adam_corrections(long long, float *c1, float *c2) { *c1 = *c2 = 1.0f; }
cudaError_t mlp_pack(const float *p, void *a, void *b, void *c, cudaStream_t s)
{
    return Launch(s, "pack").read(p).write(a).write(b).write(c).done();
}
cudaError_t mlp_cell_hist(const void *d, int, int, int, int, int, int, int, int, float, float, float *h, cudaStream_t s)
{
    return Launch(s, "cell histograms").read(d).write(h).done();
}
cudaError_t mlp_cell_features(const float *mc, const float *hist, int, float, float, const float *knots, const float4 *,
                              int, int, float, void *x, float *t, cudaStream_t s)
{
    return Launch(s, "features").read(mc).read(hist).read(knots).write(x).write(t).done();
}
cudaError_t mlp_tf_knots(const float4 *, int, float *k, cudaStream_t s) { return Launch(s, "knots").write(k).done(); }
cudaError_t mlp_learned_grid_tc(const MlpDev &, const MlpGridArgs &a, cudaStream_t s)
{
    return Launch(s, "learned grid").read(a.mc).read(a.hist).read(a.knots).write(a.dist).done();
}
cudaError_t mlp_calibrate(const float *y, const float *t, long long, float, int *, unsigned long long *, cudaStream_t s)
{
    return Launch(s, "calibrate").read(y).read(t).done();
}
float mlp_key_value(int) { return 0.0f; }
int mlp_key_of(float) { return 0; }

}  // namespace ivr
