// evp_transfer.cu -- a call's fields between the caller's host arrays and the
// slot-ordered device state.
//
// Arrays that the GPU can address (page-locked or managed memory, the whole
// range checked) are read and written by the kernels themselves, each field
// once, in the caller's order: k_upload takes a point's 29 values, skip flags
// included, and writes every place they go to (both state sets, the
// slot-ordered inputs, the constant blocks); k_download gathers the results.
// Other arrays pass through page-locked staging, once a program's calls have
// paid for it: a small call's by one copy by the host and the same kernels; a
// large call's in chunks that several host threads copy while the copy engine
// moves others to or from device staging.  Before that they go by cudaMemcpyAsync.
//
// What bounds it: the host link for large calls; for small ones it was the
// number of copies (31 up, 17 down, about 2 us each, and a dozen kernels
// and fills): 2.0k points took 190 us up and 90 us down.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "evp_internal.h"

namespace evp {

namespace {

#define CUDA_TRY(x)                                                        \
  do {                                                                     \
    cudaError_t e_ = (x);                                                  \
    if (e_ != cudaSuccess)                                                 \
      return error(e_ == cudaErrorMemoryAllocation ? EVP1D_ERR_NOMEM       \
                                                   : EVP1D_ERR_CUDA,       \
                   "%s: %s", #x, cudaGetErrorString(e_));                  \
  } while (0)

// The page-locked staging buffer, and the staged bytes of one call up to which
// the kernels go to it: one host thread fills it at about 10 GB/s, which
// overlaps with nothing; larger calls take chunks of it in turn.
constexpr size_t kPinnedStage = 8u << 20, kStagedDirect = 3u << 20;
static_assert(kStagedDirect <= kPinnedStage, "one call's staging");
// Host threads of a chunked copy: one per kThreadBytes, up to kMaxThreads (a
// thread takes 30 us to start and copies about 10 GB/s; 42 MB into fresh pages
// took 3.0, 2.5, 1.4 and 0.9 ms on 1, 2, 4 and 8 threads, and 5.9 through
// cudaMemcpyAsync's own staging).
constexpr size_t kThreadBytes = 2u << 20;
constexpr int kMaxThreads = 8;

// Bytes of one call up to which the kernels go to addressable host arrays
// themselves.  They move about 40 GB/s over the host link where
// cudaMemcpyAsync's copy engine moves 55, which pays for its 31 (17) copies of
// 3 us each only in larger calls, us up and down by the kernels and by copies:
// 74k points 406, 240 and 537, 268; 124k 675, 370 and 731, 398; 296k 1765,
// 1085 and 1629, 829.  Calls with an index map (2D arrays: only the list's
// cells travel) always go direct.
constexpr size_t kDirectUp = 40u << 20, kDirectDown = 20u << 20;

constexpr int kThreads = 128;

struct UploadArgs {
  int na, navel, nslots, nuv;
  const int32_t *slot_of_point, *tile_of_quad, *tile_off;
  const int32_t *map_f, *map_uv;  // null: the point itself
  bool mask, zero_halo;
  double rhow;
  const double *in[12], *stress[12];
  const double *u, *v, *uinit, *vinit, *strintx, *strinty, *Cb;
  const int32_t *skT, *skU;
  // destinations, by slot
  double *dyn[kNumDyn];
  double *s0[12], *s1[12], *u0, *u1, *v0, *v1, *o_strintx, *o_strinty, *o_Cb, *str[8];
  const uint32_t *lnb, *lcor;
  uint8_t *flags;
  uint32_t *meta;
  double *cblk;
  int *cflags;
};

__global__ void __launch_bounds__(kThreads) k_upload(UploadArgs a) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i < a.nuv) {
#pragma unroll
    for (int k = 0; k < 8; k++) a.str[k][i] = 0.0;
  }
  if (i >= a.navel) return;
  if (i >= a.na) {  // the reference's halo slots
    const int s = a.nslots + (i - a.na);
    double u = 0.0, v = 0.0;
    if (!a.zero_halo) {
      const int c = a.map_uv ? a.map_uv[i] : i;
      u = a.u[c];
      v = a.v[c];
    }
    a.u0[s] = a.u1[s] = u;
    a.v0[s] = a.v1[s] = v;
    return;
  }
  const int s = a.slot_of_point[i];
  const int c = a.map_f ? a.map_f[i] : i;
  const int cu = a.map_uv ? a.map_uv[i] : c;
  double in[12], st[12];
#pragma unroll
  for (int k = 0; k < 12; k++) in[k] = a.in[k][c];
#pragma unroll
  for (int k = 0; k < 12; k++) st[k] = a.stress[k][c];
  const double u = a.u[cu], v = a.v[cu];
  const double ui = a.uinit ? a.uinit[c] : u, vi = a.vinit ? a.vinit[c] : v;
  const double sx = a.strintx[c], sy = a.strinty[c], cb = a.Cb[c];
  const int32_t mt = a.skT[c], mu = a.skU[c];
  const uint32_t fl = ((mt != 0) != a.mask ? kSkipT : 0u) | ((mu != 0) != a.mask ? kSkipU : 0u);
  const uint32_t meta = a.lnb[s] | fl << 30;
  a.flags[s] = (uint8_t)fl;
  a.meta[s] = meta;
  const double kv = drag_factor(in[kAiu], a.rhow, in[kCw]);
#pragma unroll
  for (int k = 0; k < 12; k++) {
    a.dyn[k][s] = in[k];
    a.s0[k][s] = st[k];
    a.s1[k][s] = st[k];
  }
  a.dyn[kUinit][s] = ui;
  a.dyn[kVinit][s] = vi;
  a.dyn[kKvrel][s] = kv;
  a.u0[s] = a.u1[s] = u;
  a.v0[s] = a.v1[s] = v;
  a.o_strintx[s] = sx;
  a.o_strinty[s] = sy;
  a.o_Cb[s] = cb;
  // the tile's constant block (launch_const_blocks), without the geometry
  const int t = a.tile_of_quad[s >> 2];
  double *blk = a.cblk + (size_t)t * kConstFields * kConstTileSlots + (s - a.tile_off[t]);
  const unsigned long long su = (unsigned long long)__double_as_longlong(ui) >> 63;
  const unsigned long long sv = (unsigned long long)__double_as_longlong(vi) >> 63;
  auto put = [&](int f, double x) { blk[(size_t)f * kConstTileSlots] = x; };
  put(6, in[kStrength]);
  put(7, __longlong_as_double((long long)((unsigned long long)meta |
                                          ((unsigned long long)a.lcor[s] << 32) | su << 62 |
                                          sv << 63)));
  put(8, kv);
#pragma unroll
  for (int k = kUocn; k <= kFm; k++) put(9 + (k - kUocn), in[k]);
  put(18, in[kTbu]);
  put(19, ui);
  put(20, vi);
  const int bad = (__double_as_longlong(in[kTbu]) != 0 ? 1 : 0) |
                  (!isfinite(ui) || !isfinite(vi) ? 2 : 0);
  if (bad) atomicOr(a.cflags, bad);
}
static_assert(kConstStressFields == 8 && kConstFields == 21 && kFm - kUocn == 7,
              "constant block layout");

struct DownloadArgs {
  int na, navel, nslots;
  const int32_t *slot_of_point;
  const int32_t *map_f, *map_uv;
  const double *s[12], *u, *v, *strintx, *strinty, *Cb, *str[8];
  double *o_s[12], *o_u, *o_v, *o_strintx, *o_strinty, *o_Cb, *o_str[8];  // null: not wanted
  const int *err;
};

__global__ void __launch_bounds__(kThreads) k_download(DownloadArgs a) {
  // a wait that ran out: the results are not valid, the caller's arrays stay
  if (*a.err) return;
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= a.navel) return;
  const int s = i < a.na ? a.slot_of_point[i] : a.nslots + (i - a.na);
  const int cu = a.map_uv ? a.map_uv[i] : i;
#pragma unroll
  for (int k = 0; k < 8; k++)
    if (a.o_str[k]) a.o_str[k][cu] = a.str[k][s];
  if (i >= a.na) return;  // halo velocities are never written
  const int c = a.map_f ? a.map_f[i] : i;
  const int cv = a.map_uv ? cu : c;
#pragma unroll
  for (int k = 0; k < 12; k++)
    if (a.o_s[k]) a.o_s[k][c] = a.s[k][s];
  if (a.o_u) a.o_u[cv] = a.u[s];
  if (a.o_v) a.o_v[cv] = a.v[s];
  if (a.o_strintx) a.o_strintx[c] = a.strintx[s];
  if (a.o_strinty) a.o_strinty[c] = a.strinty[s];
  if (a.o_Cb) a.o_Cb[c] = a.Cb[s];
}

// The driver's range query: where an address is page-locked, managed or device
// memory, the allocation around it.
using PtrAttrs = int (*)(unsigned, int *, void **, unsigned long long);

PtrAttrs ptr_attrs() {
  static const PtrAttrs f = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<PtrAttrs>(p);
  }();
  return f;
}

// One page-locked block: kWords error words, then the staging buffer.
// Page-locking it takes 4 to 10 ms (one page: 2.5), during which no other CUDA
// call of the process gets on, so a program's first calls go without it: copies
// by cudaMemcpyAsync from and to ordinary memory, each about 5 us dearer (and 5
// us per 128 KB), and the block comes once they would have paid for it.  First
// transfers of a handle in ordinary memory, 64x48 and 400x300, ms: 4 and 9 with
// the block, 0.8 and 2.7 without; a handle's creation 7 and 4 ms at 64x48.
struct PinnedPool {
  static constexpr int kWords = 1024;
  static constexpr size_t kPays = 1000, kItem = 128u << 10;
  std::mutex m;
  unsigned gen = 0;  // counts the blocks: handles of an older one hold nothing
  int refs = 0;
  size_t owed = 0;   // copies made without the block, in units of 5 us
  char *block = nullptr;
  bool used[kWords] = {};
  bool lent = false;

  int *words() { return reinterpret_cast<int *>(block); }
  char *stage() { return block + kWords * sizeof(int); }
  // Whether the block is there, for a call that would make `copies` copies of
  // `bytes` in all without it.
  bool ready(size_t copies, size_t bytes) {
    if (block || refs == 0) return block != nullptr;
    owed += copies + bytes / kItem;
    if (owed < kPays) return false;
    owed = 0;
    void *p = nullptr;
    if (cudaHostAlloc(&p, kWords * sizeof(int) + kPinnedStage, cudaHostAllocPortable) !=
        cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    block = static_cast<char *>(p);
    return true;
  }
  void forget() {
    gen++;
    refs = 0;
    owed = 0;
    block = nullptr;
    lent = false;
    for (bool &u : used) u = false;
  }
};
PinnedPool &pool() {
  static PinnedPool p;
  return p;
}

// The staging buffer for a call of so many copies and bytes, or null where it
// does not pay yet or while another call has it (the caller then takes device
// staging).
char *borrow_stage(size_t copies, size_t bytes) {
  PinnedPool &p = pool();
  std::lock_guard<std::mutex> lock(p.m);
  if (p.lent || !p.ready(copies, bytes)) return nullptr;
  p.lent = true;
  return p.stage();
}

void return_stage() {
  PinnedPool &p = pool();
  std::lock_guard<std::mutex> lock(p.m);
  p.lent = false;
}

}  // namespace

void pinned_hold(DeviceProblem *d) {
  PinnedPool &p = pool();
  std::lock_guard<std::mutex> lock(p.m);
  // A reset of the device (cudaDeviceReset) takes the memory away from under
  // handles that were not finalized: the pool starts anew.
  cudaPointerAttributes at;
  if (p.block && (cudaPointerGetAttributes(&at, p.block) != cudaSuccess ||
                  at.type != cudaMemoryTypeHost)) {
    cudaGetLastError();
    p.forget();
  }
  p.refs++;
  d->pins = true;
  d->pin_gen = p.gen;
}

void pinned_release(DeviceProblem *d) {
  if (!d->pins) return;
  PinnedPool &p = pool();
  std::lock_guard<std::mutex> lock(p.m);
  d->pins = false;
  if (d->pin_gen != p.gen) return;
  if (d->err_host) p.used[d->err_host - p.words()] = false;
  d->err_host = nullptr;
  if (--p.refs > 0) return;
  if (p.block) cudaFreeHost(p.block);
  p.forget();
}

int *pinned_word(DeviceProblem *d) {
  if (d->err_host || !d->pins) return d->err_host;
  PinnedPool &p = pool();
  std::lock_guard<std::mutex> lock(p.m);
  if (d->pin_gen != p.gen || !p.ready(1, sizeof(int))) return nullptr;
  for (int k = 0; k < PinnedPool::kWords && !d->err_host; k++)
    if (!p.used[k]) {
      p.used[k] = true;
      d->err_host = p.words() + k;
    }
  return d->err_host;
}

namespace {

// Whose memory a caller's array is: the host's own (pageable, or not wholly
// registered), the GPU's to address as well, or a device's alone, which no host
// code may touch (cudaMemcpyAsync copies it).
enum HostKind { kPageable, kAddressable, kDeviceOnly };

HostKind host_kind(const void *p, size_t bytes, size_t align, void **dev) {
  PtrAttrs query = ptr_attrs();
  if (!query || !p || bytes == 0) return kPageable;
  // CUpointer_attribute: MEMORY_TYPE 2, DEVICE_POINTER 3, IS_MANAGED 8,
  // RANGE_START_ADDR 11, RANGE_SIZE 12
  int what[5] = {2, 3, 8, 11, 12};
  unsigned type = 0, managed = 0;
  unsigned long long dptr = 0, start = 0;
  size_t size = 0;
  void *out[5] = {&type, &dptr, &managed, &start, &size};
  const unsigned long long at = (unsigned long long)(uintptr_t)p;
  if (query(5, what, out, at) != 0) return kPageable;
  constexpr unsigned kHost = 1, kDevice = 2, kArray = 3;  // CUmemorytype
  if ((type == kDevice || type == kArray) && !managed) return kDeviceOnly;
  if (!(type == kHost || managed) || dptr == 0 || start == 0) return kPageable;
  // the range query gives the allocation in the address space it is asked in
  // (host addresses of page-locked memory equal its device addresses); an
  // array that only begins in registered memory is not addressable
  const unsigned long long base = at >= start && at < start + size ? at : dptr;
  if (base < start || bytes > size || base - start > size - bytes) return kPageable;
  if (dptr % align) return kPageable;
  *dev = reinterpret_cast<void *>((uintptr_t)dptr);
  return kAddressable;
}

// One array between host memory and device staging.
struct CopyItem {
  char *host, *dev;
  size_t bytes;
  HostKind kind;
};

// Pageable items through `stage` (kPinnedStage bytes) in chunks, each host
// thread with two halves of its own share of it.  Up: the copies are queued on
// the stream, and complete, on return; down: the results are in host memory.
cudaError_t copy_chunked(const std::vector<CopyItem> &items, bool up, char *stage, int device,
                         cudaStream_t st) {
  size_t total = 0;
  for (const CopyItem &it : items) total += it.bytes;
  const unsigned hw = std::thread::hardware_concurrency();
  int nt = (int)std::min<size_t>(kMaxThreads, total / kThreadBytes);
  if (hw > 0 && nt > (int)hw) nt = (int)hw;
  if (nt < 1) nt = 1;
  const size_t half = (kPinnedStage / nt / 2) & ~size_t(4095);
  std::vector<CopyItem> chunks;
  for (const CopyItem &it : items)
    for (size_t o = 0; o < it.bytes; o += half)
      chunks.push_back({it.host + o, it.dev + o, std::min(half, it.bytes - o), it.kind});
  std::atomic<size_t> next{0};
  std::atomic<int> failed{(int)cudaSuccess};
  auto work = [&](int w) {
    auto check = [&](cudaError_t e) {
      int none = (int)cudaSuccess;
      if (e != cudaSuccess) failed.compare_exchange_strong(none, (int)e);
      return e == cudaSuccess;
    };
    char *buf[2] = {stage + (size_t)w * 2 * half, stage + ((size_t)w * 2 + 1) * half};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    const CopyItem *busy[2] = {nullptr, nullptr};
    bool ok = check(cudaSetDevice(device)) &&
              check(cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming)) &&
              check(cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming));
    // the copy queued on half b has ended; down: its chunk goes to the caller
    auto drain = [&](int b) {
      if (!busy[b]) return true;
      const CopyItem *c = busy[b];
      busy[b] = nullptr;
      if (!check(cudaEventSynchronize(ev[b]))) return false;
      if (!up) memcpy(c->host, buf[b], c->bytes);
      return true;
    };
    int b = 0;
    while (ok && failed.load() == (int)cudaSuccess) {
      const size_t k = next.fetch_add(1);
      if (k >= chunks.size()) break;
      const CopyItem &c = chunks[k];
      ok = drain(b);
      if (!ok) break;
      if (up) memcpy(buf[b], c.host, c.bytes);
      ok = check(up ? cudaMemcpyAsync(c.dev, buf[b], c.bytes, cudaMemcpyHostToDevice, st)
                    : cudaMemcpyAsync(buf[b], c.dev, c.bytes, cudaMemcpyDeviceToHost, st)) &&
           check(cudaEventRecord(ev[b], st));
      if (!ok) break;
      busy[b] = &c;
      b ^= 1;
    }
    if (ok) ok = drain(b) && drain(b ^ 1);
    if (!ok) cudaStreamSynchronize(st);  // nothing may still be reading the halves
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
  };
  std::vector<std::thread> threads;
  try {
    threads.reserve((size_t)nt);
    for (int w = 1; w < nt; w++) threads.emplace_back(work, w);
  } catch (...) {
    // fewer threads than wanted: the chunks are taken by those there are
  }
  work(0);
  for (std::thread &t : threads) t.join();
  return (cudaError_t)failed.load();
}

// One item by the copy engine's own call.  It refuses ordinary memory of which
// a part is registered: that goes by way of other memory.
cudaError_t copy_plain(const CopyItem &it, bool up, cudaStream_t st) {
  cudaError_t e = up ? cudaMemcpyAsync(it.dev, it.host, it.bytes, cudaMemcpyHostToDevice, st)
                     : cudaMemcpyAsync(it.host, it.dev, it.bytes, cudaMemcpyDeviceToHost, st);
  if (e != cudaErrorInvalidValue || it.kind != kPageable) return e;
  cudaGetLastError();
  std::unique_ptr<char[]> way(new (std::nothrow) char[it.bytes]);
  if (!way) return cudaErrorMemoryAllocation;
  if (up) memcpy(way.get(), it.host, it.bytes);
  e = up ? cudaMemcpyAsync(it.dev, way.get(), it.bytes, cudaMemcpyHostToDevice, st)
         : cudaMemcpyAsync(way.get(), it.dev, it.bytes, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && !up) memcpy(it.host, way.get(), it.bytes);
  return e;
}

// Every item: pageable ones in chunks where the staging buffer is free and
// they are large, the others by the copy engine's own call.  Up: queued on
// return, and pageable memory is no longer read; down: queued (pageable:
// complete).
cudaError_t copy_items(const std::vector<CopyItem> &items, bool up, int device, cudaStream_t st) {
  std::vector<CopyItem> own;
  size_t total = 0;
  for (const CopyItem &it : items) {
    if (it.kind == kPageable) {
      own.push_back(it);
      total += it.bytes;
      continue;
    }
    const cudaError_t e = copy_plain(it, up, st);
    if (e != cudaSuccess) return e;
  }
  if (own.empty()) return cudaSuccess;
  struct Loan {
    char *stage;
    ~Loan() {
      if (stage) return_stage();
    }
  } loan{total >= kThreadBytes ? borrow_stage(own.size(), total) : nullptr};
  if (loan.stage) return copy_chunked(own, up, loan.stage, device, st);
  for (const CopyItem &it : own) {
    const cudaError_t e = copy_plain(it, up, st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

bool device_view(const void *p, size_t bytes, size_t align, void **dev) {
  return host_kind(p, bytes, align, dev) == kAddressable;
}

namespace {

// Where each array of a call is for the kernels.
struct Placer {
  size_t direct_limit;
  explicit Placer(size_t limit) : direct_limit(limit) {}
  ~Placer() {
    if (pinned) return_stage();
  }
  Placer(const Placer &) = delete;
  Placer &operator=(const Placer &) = delete;
  struct Item {
    const void *host;
    void *stage;  // device staging of the array
    size_t bytes;
    void **dev;   // the pointer the kernels get
    HostKind kind;
    size_t off = 0;
  };
  std::vector<Item> staged, direct;
  size_t total = 0, direct_total = 0;
  bool pinned = false;
  bool foreign = false;  // a device's own memory among the arrays

  // dev: device address for the kernels, at once where the GPU can address the
  // array, else set by place().  `fixed`: an array its map makes direct.
  void add(const void *host, size_t bytes, size_t align, void *stage, void **dev,
           bool fixed = false) {
    const HostKind kind = host_kind(host, bytes, align, dev);
    if (kind == kAddressable) {
      if (!fixed) {
        direct.push_back({host, stage, bytes, dev, kind});
        direct_total += bytes;
      }
    } else {
      foreign = foreign || kind == kDeviceOnly;
      stage_it({host, stage, bytes, dev, kind});
    }
  }
  void stage_it(Item it) {
    *it.dev = it.stage;
    it.off = total;
    total += (it.bytes + 255) & ~size_t(255);
    staged.push_back(it);
  }
  // Page-locked staging for the staged arrays, where they are small; the copy
  // engine for addressable ones, where they are many.
  void place() {
    if (direct_total > direct_limit) {
      for (const Item &it : direct) stage_it(it);
      return;
    }
    if (staged.empty() || foreign || total > kStagedDirect) return;
    char *base = borrow_stage(staged.size(), total);
    if (!base) return;
    pinned = true;
    for (Item &it : staged) *it.dev = base + it.off;
  }
  std::vector<CopyItem> copies() const {
    std::vector<CopyItem> c;
    for (const Item &it : staged)
      c.push_back({(char *)it.host, (char *)it.stage, it.bytes, it.kind});
    return c;
  }
};

// The lists of a call's arrays could not grow (no exception may leave a C entry
// point).  The copies queued so far end first.
int no_memory(DeviceProblem *d) {
  cudaStreamSynchronize(d->stream);
  return error(EVP1D_ERR_NOMEM, "out of memory");
}

}  // namespace

int problem_upload(DeviceProblem *d, const UploadFields &f, double rhow, bool wait) try {
  if (d->na == 0) return EVP1D_OK;
  cudaStream_t st = d->stream;
  UploadArgs a;
  a.na = d->na;
  a.navel = d->navel;
  a.nslots = d->nslots;
  a.nuv = d->nuv;
  a.slot_of_point = d->slot_of_point;
  a.tile_of_quad = d->tile_of_quad;
  a.tile_off = d->tile_off;
  a.map_f = f.map_f;
  a.map_uv = f.map_uv;
  a.mask = f.mask;
  a.zero_halo = f.zero_halo;
  a.rhow = rhow;
  Placer P(kDirectUp);
  const size_t bf = f.n_f * sizeof(double), bu = f.n_uv * sizeof(double);
  int slot = 0;
  auto take = [&](const double *host, size_t bytes, const double **dev, bool fixed = false) {
    double *stage = f.stage + (size_t)(slot++) * f.stage_step;
    P.add(host, bytes, sizeof(double), stage, (void **)dev, fixed);
  };
  for (int k = 0; k < 12; k++) take(f.in[k], bf, &a.in[k]);
  for (int k = 0; k < 12; k++) take(f.stress[k], bf, &a.stress[k]);
  take(f.strintx, bf, &a.strintx);
  take(f.strinty, bf, &a.strinty);
  take(f.Cb, bf, &a.Cb);
  take(f.u, bu, &a.u, f.map_uv != nullptr);
  take(f.v, bu, &a.v, f.map_uv != nullptr);
  a.uinit = a.vinit = nullptr;
  if (f.uinit) take(f.uinit, bf, &a.uinit);
  if (f.vinit) take(f.vinit, bf, &a.vinit);
  const size_t bi = f.n_f * sizeof(int32_t);
  P.add(f.skT, bi, sizeof(int32_t), f.istage, (void **)&a.skT);
  P.add(f.skU, bi, sizeof(int32_t), f.istage + f.n_f, (void **)&a.skU);
  // (2D arrays: the device staging keeps the cells outside the list for the
  // way back)
  if (!f.map_f) P.place();
  if (P.pinned)
    for (const Placer::Item &it : P.staged) memcpy(*it.dev, it.host, it.bytes);
  else
    CUDA_TRY(copy_items(P.copies(), true, d->device, st));
  for (int k = 0; k < kNumDyn; k++) a.dyn[k] = d->dyn[k];
  for (int k = 0; k < 12; k++) {
    a.s0[k] = d->stress[0][k];
    a.s1[k] = d->stress[1][k];
  }
  a.u0 = d->u[0];
  a.u1 = d->u[1];
  a.v0 = d->v[0];
  a.v1 = d->v[1];
  a.o_strintx = d->strintx;
  a.o_strinty = d->strinty;
  a.o_Cb = d->Cb;
  for (int k = 0; k < 8; k++) a.str[k] = d->str[k];
  a.lnb = d->lnb;
  a.lcor = d->lcor;
  a.flags = d->flags;
  a.meta = d->meta;
  a.cblk = d->cblk;
  a.cflags = d->cflags;
  CUDA_TRY(cudaMemsetAsync(d->cflags, 0, sizeof(int), st));
  const int n = d->nuv > d->navel ? d->nuv : d->navel;
  k_upload<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(a);
  CUDA_TRY(cudaGetLastError());
  // (the borrowed staging goes back when this returns)
  if (wait || P.pinned) CUDA_TRY(cudaStreamSynchronize(st));
  d->cur = 0;
  return EVP1D_OK;
} catch (const std::bad_alloc &) {
  return no_memory(d);
}

int problem_download(DeviceProblem *d, const DownloadFields &f, int *code) try {
  *code = 0;
  if (d->na == 0) return EVP1D_OK;
  cudaStream_t st = d->stream;
  DownloadArgs a;
  a.na = d->na;
  a.navel = d->navel;
  a.nslots = d->nslots;
  a.slot_of_point = d->slot_of_point;
  a.map_f = f.map_f;
  a.map_uv = f.map_uv;
  a.err = d->err;
  const int c = d->cur;
  Placer P(kDirectDown);
  auto give = [&](const double *src, double *host, size_t elems, const double **from, double **to,
                  int at, bool fixed = false) {
    *from = src;
    *to = nullptr;
    double *stage = f.stage + (size_t)at * f.stage_step;
    if (host) P.add(host, elems * sizeof(double), sizeof(double), stage, (void **)to, fixed);
  };
  const bool fixed = f.map_uv != nullptr;
  for (int k = 0; k < 12; k++) give(d->stress[c][k], f.stress[k], f.n_f, &a.s[k], &a.o_s[k], 12 + k);
  give(d->strintx, f.strintx, f.n_f, &a.strintx, &a.o_strintx, 24);
  give(d->strinty, f.strinty, f.n_f, &a.strinty, &a.o_strinty, 25);
  give(d->Cb, f.Cb, f.n_f, &a.Cb, &a.o_Cb, 26);
  give(d->u[c], f.u, f.n_u, &a.u, &a.o_u, 27, fixed);
  give(d->v[c], f.v, f.n_u, &a.v, &a.o_v, 28, fixed);
  for (int k = 0; k < 8; k++)
    give(d->str[k], f.str[k], f.n_str, &a.str[k], &a.o_str[k], k, fixed);
  // Staged arrays of a 2D call hold the caller's values of the other cells in
  // the device staging since the upload: they stay there.
  if (!f.map_f) P.place();
  if (!P.staged.empty() && !P.pinned) {
    // nothing of the caller's is overwritten after a wait that ran out
    const int rc = problem_take_error(d, code);
    if (rc != EVP1D_OK || *code) return rc;
  }
  k_download<<<(d->navel + kThreads - 1) / kThreads, kThreads, 0, st>>>(a);
  CUDA_TRY(cudaGetLastError());
  if (!P.pinned) CUDA_TRY(copy_items(P.copies(), false, d->device, st));
  const int rc = problem_take_error(d, code);  // waits for the stream
  if (rc != EVP1D_OK || *code) return rc;
  if (P.pinned)
    for (const Placer::Item &it : P.staged) memcpy(const_cast<void *>(it.host), *it.dev, it.bytes);
  return EVP1D_OK;
} catch (const std::bad_alloc &) {
  return no_memory(d);
}

int problem_gather_to_host(DeviceProblem *d, int n, const double *const *src,
                           double *const *host) try {
  const size_t bytes = (size_t)d->na * sizeof(double);
  cudaStream_t st = d->stream;
  for (int at = 0; at < n; at += kMaxBatch) {
    const int m = std::min(kMaxBatch, n - at);
    Placer P(kDirectDown);
    PermBatch b;
    b.n = m;
    void *to[kMaxBatch];
    for (int k = 0; k < m; k++) {
      b.src[k] = src[at + k];
      P.add(host[at + k], bytes, sizeof(double),
            d->stage + (size_t)k * (size_t)(d->navel > 0 ? d->navel : 1), &to[k]);
    }
    P.place();
    for (int k = 0; k < m; k++) b.dst[k] = static_cast<double *>(to[k]);
    launch_gather(b, d->na, d->slot_of_point, st);
    CUDA_TRY(cudaGetLastError());
    if (!P.pinned) CUDA_TRY(copy_items(P.copies(), false, d->device, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    if (P.pinned)
      for (const Placer::Item &it : P.staged)
        memcpy(const_cast<void *>(it.host), *it.dev, it.bytes);
  }
  return EVP1D_OK;
} catch (const std::bad_alloc &) {
  return no_memory(d);
}

}  // namespace evp
