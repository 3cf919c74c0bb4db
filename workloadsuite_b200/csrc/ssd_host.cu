// Host-buffer entry point: the SSD forward for callers whose tensors live in
// host memory.  Each batch entry is cut along the SEQUENCE into chunks of a few
// thousand tokens: a chunk of X, Y, B, C, A, dt is one contiguous block of host
// memory (plain 1-D copies at full PCIe rate), and the scan carries over from
// chunk to chunk through the fp32 state, which stays on the device.  The call
// is a three-stage pipeline over chunks: host->device copies of chunk i+1,
// kernels of chunk i and device->host copy of chunk i-1 run on three streams
// and overlap (PCIe is full duplex).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "ssd_common.cuh"

namespace {

constexpr int kSlots = 4;
constexpr int kMaxDevices = 64;

// Streams and events of the host-buffer pipeline, created on first use per device and kept.
struct Pipe {
  cudaStream_t st_in = nullptr, st_run = nullptr, st_out = nullptr;
  std::vector<cudaEvent_t> events;
};
Pipe g_pipes[kMaxDevices];
std::mutex g_pipes_mu[kMaxDevices];

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
int esize(int dtype) { return dtype == SSD_DTYPE_F32 ? 4 : 2; }
int gcd_int(int a, int b) { return b == 0 ? a : gcd_int(b, a % b); }

struct Plan {
  int tokens;      // tokens per chunk (the last chunk of a sequence may be shorter)
  int nchunks;     // chunks per batch entry
  int group;       // batch entries per chunk (> 1 only when a whole entry is much smaller than a chunk)
  int set_entries; // batch entries whose B, C, A, dt (and entering state) travel together
  size_t x_bytes, a_bytes, dt_bytes, bc_bytes, ws_bytes, st_bytes, enter_bytes;   // a, dt, bc, enter: one set
  size_t slot_bytes, set_bytes, ldall_bytes, total_bytes;
  int nslices;
};

bool basic_ok(const SsdArgs* a) {
  return a && a->batch > 0 && a->seqlen > 0 && a->nheads > 0 && a->headdim > 0 && a->dstate > 0 && a->ngroups > 0 &&
         a->nheads % a->ngroups == 0 && a->chunk > 0 && a->seqlen % a->chunk == 0 &&
         (a->dtype == SSD_DTYPE_F32 || a->dtype == SSD_DTYPE_F16 || a->dtype == SSD_DTYPE_BF16);
}

// Arguments of the forward over one chunk of one batch entry (pointers are filled in by the caller).
void chunk_args(const SsdArgs* a, int tokens, int entries, SsdArgs* s) {
  *s = *a;
  s->batch = entries;
  s->seqlen = tokens;
  s->nsegments = 0;
  s->status = nullptr;   // (the pipeline points it at the status word inside its device scratch)
  s->D = nullptr;
  s->Z = nullptr;
  // `a` holds HOST pointers: kernel choice and scratch size must follow the device buffers, which are
  // 256-byte aligned, so the tensor pointers are cleared here (a shape query) and set by the pipeline
  s->X = nullptr; s->A = nullptr; s->B = nullptr; s->C = nullptr; s->Y = nullptr;
  s->initial_state = nullptr; s->final_state = nullptr; s->final_logdecay = nullptr;
  s->workspace = nullptr; s->workspace_bytes = 0;
  // the chunk's tensors are contiguous in the device buffers (kernel choice and scratch size depend on the strides)
  const int64_t h = a->nheads, p = a->headdim, g = a->ngroups, n = a->dstate;
  const int64_t xs[3] = {tokens * h * p, h * p, p}, as[3] = {tokens * h, h, 1}, bs[3] = {tokens * g * n, g * n, n};
  for (int k = 0; k < 3; ++k) {
    s->x_stride[k] = xs[k]; s->y_stride[k] = xs[k]; s->a_stride[k] = as[k]; s->dt_stride[k] = as[k];
    s->b_stride[k] = bs[k]; s->c_stride[k] = bs[k];
  }
}

struct Slice {
  int bi, nb, ci, t0, tokens;   // nb batch entries from bi on
  bool first, last;
  int set, set_bi, set_nb;      // ordinal of the set that the entries belong to, and its entries
};

// A copy costs some 20 us beside one in the other direction, whatever its size: what is small next to X goes in few
// copies, several batch entries at a time, only the first set being as small as the first chunk.
void make_sets(std::vector<Slice>& slices, int set_entries) {
  int set = -1, begin = 0, end = 0;
  for (size_t i = 0; i < slices.size(); ++i) {
    if (slices[i].bi + slices[i].nb > end) {
      ++set;
      begin = slices[i].bi;
      end = begin + slices[i].nb;
      for (size_t k = i + 1; set > 0 && k < slices.size() && slices[k].bi + slices[k].nb - begin <= set_entries; ++k)
        end = slices[k].bi + slices[k].nb;
    }
    slices[i].set = set;
    slices[i].set_bi = begin;
    slices[i].set_nb = end - begin;
  }
}

// From 64 MiB of X on the link is busy for long enough that what a copy costs of its own (some 20 us) matters less than how much
// of the last chunk is still to come back when the last input is in: chunks of an eighth of the whole, and what is small next to
// X with its own chunk.  Below, fewer and larger ones.  16 entries of 10.5 MB: 4.14 ms so, 4.46 in quarters with sets of four
// entries; 16 of 12.6 MB: 5.25 and 5.54; but 4 entries of 6.3 MB: 0.99 and 0.86, 64 of 0.13 MB: 0.49 and 0.40.
bool is_large(const SsdArgs* a) {
  return (int64_t)a->nheads * a->headdim * esize(a->dtype) * a->seqlen >= (((int64_t)64 << 20) + a->batch - 1) / a->batch;
}

// Pieces of 1/4, 1/4, 1/2 of `regular` (`fine`: 1/8, 1/8, 1/4, 1/2; multiples of `unit`), as far as they fit into `left` with
// `keep` to spare and are worth a copy of their own (at least `least`).
std::vector<int> ramp(int regular, int unit, int least, int keep, int* left, bool fine) {
  std::vector<int> pieces;
  const std::vector<int> div = fine ? std::vector<int>{8, 8, 4, 2} : std::vector<int>{4, 4, 2};
  for (int d : div) {
    const int len = regular / d / unit * unit;
    if (len >= std::max(1, least) && *left - len >= keep) {
      pieces.push_back(len);
      *left -= len;
    }
  }
  return pieces;
}

// The chunks of all batch entries in order.  They open and close with a ramp of smaller ones, so that the device->host
// stream starts early and the host->device stream ends late: the two directions then overlap for all but a fraction of a
// chunk (also where a chunk is a whole batch entry; or several, where the whole is not large).
std::vector<Slice> make_slices(const SsdArgs* host, int tokens_per_chunk, int group, int set_entries) {
  std::vector<Slice> slices;
  const int b = host->batch, s = host->seqlen;
  const int64_t row = (int64_t)host->nheads * host->headdim * esize(host->dtype);
  const bool large = is_large(host);
  constexpr int64_t kLeastBytes = 384 << 10;   // of X in a piece: a copy, a launch and two event waits cost some 10 us
  int unit = host->chunk / gcd_int(host->chunk, 128) * 128;
  if (s % unit != 0) unit = host->chunk;
  if (group > 1) {
    const int least = (int)std::min<int64_t>(b, (kLeastBytes + row * s - 1) / (row * s));
    int left = b;
    std::vector<int> sizes, tail;
    if (!large) {
      sizes = ramp(group, 1, least, std::min(b, 2 * group) / 2, &left, false);
      tail = ramp(group, 1, least, 0, &left, false);
    }
    for (; left > 0; left -= std::min(group, left)) sizes.push_back(std::min(group, left));
    sizes.insert(sizes.end(), tail.rbegin(), tail.rend());
    int bi = 0;
    for (int nb : sizes) {
      slices.push_back({bi, nb, 0, 0, s, true, true, 0, 0, 0});
      bi += nb;
    }
    make_sets(slices, set_entries);
    return slices;
  }
  const int least = (int)std::min<int64_t>(s, (kLeastBytes + row - 1) / row);
  for (int bi = 0; bi < b; ++bi) {
    int left = s;
    std::vector<int> lens, tail;
    const int keep = large ? tokens_per_chunk : b == 1 ? std::min(s, 2 * tokens_per_chunk) / 2 : 0;
    if (bi == 0) lens = ramp(tokens_per_chunk, unit, least, keep, &left, large);
    if (bi == b - 1) tail = ramp(tokens_per_chunk, unit, least, large ? tokens_per_chunk : 0, &left, large);
    while (left > 0) { const int len = std::min(tokens_per_chunk, left); lens.push_back(len); left -= len; }
    lens.insert(lens.end(), tail.rbegin(), tail.rend());   // the smallest last
    int t0 = 0;
    for (size_t k = 0; k < lens.size(); ++k) {
      slices.push_back({bi, 1, (int)k, t0, lens[k], k == 0, k + 1 == lens.size(), 0, 0, 0});
      t0 += lens[k];
    }
  }
  make_sets(slices, set_entries);
  return slices;
}

Plan make_plan(const SsdArgs* a) {
  Plan pl{};
  const int e = esize(a->dtype);
  // chunk length: a multiple of the caller's chunk and of the tensor-core tile (128) when the sequence allows,
  // sized so that the X chunk is at most 48 MiB (measured on the 2.7B layer shape, 84 MB of X per batch entry: two chunks
  // of 42 MB per entry 8.5 ms, chunks of 24 / 28 / 56 / 84 MB 8.9 / 9.0 / 9.1 / 9.0 ms; with 8 MiB chunks the copies
  // in both directions together reach 78 GB/s, with 24 MiB and more 82-86 GB/s), and an eighth of the whole, or a quarter, where
  // that is less (is_large): beside copies in the other direction every copy costs some 20 us of its own (50 MB each way take
  // 1.05 ms in one piece, 1.2 in 8, 1.4 in 16, 1.65 in 32)
  int unit = a->chunk / gcd_int(a->chunk, 128) * 128;
  if (a->seqlen % unit != 0) unit = a->chunk;
  const size_t per_token = (size_t)a->nheads * a->headdim * e;
  const size_t total = per_token * a->seqlen * a->batch;
  const bool large = is_large(a);
  const size_t cap = std::max<size_t>((size_t)1 << 20, std::min<size_t>((size_t)48 << 20, total / (large ? 8 : 4)));
  // ... and a batch entry is cut into equal chunks (no short remainder chunk at the end of every entry)
  long long tokens = (long long)(cap / per_token) / unit * unit;
  tokens = std::max<long long>(unit, std::min<long long>(tokens, a->seqlen));
  {
    const long long pieces = (a->seqlen + tokens - 1) / tokens;
    const long long even = ((a->seqlen + pieces - 1) / pieces + unit - 1) / unit * unit;
    tokens = std::max<long long>(unit, std::min<long long>(even, tokens));
  }
  pl.tokens = (int)tokens;
  pl.nchunks = (a->seqlen + pl.tokens - 1) / pl.tokens;
  // short sequences: several whole batch entries (contiguous in host memory) travel and run as one chunk
  const size_t per_entry = per_token * a->seqlen;
  pl.group = 1;
  if (pl.nchunks == 1 && a->batch > 1 && per_entry * 2 <= cap)
    pl.group = (int)std::min<size_t>((size_t)a->batch, cap / per_entry);
  const size_t k = (size_t)pl.group;
  pl.x_bytes = align_up(per_token * pl.tokens * k, 256);
  const size_t entry_a = (size_t)a->seqlen * a->nheads * 4, entry_dt = a->dt ? (size_t)a->seqlen * a->nheads * e : 0;
  const size_t entry_bc = (size_t)a->seqlen * a->ngroups * a->dstate * e;
  const size_t entry_st = (size_t)a->nheads * a->dstate * a->headdim * 4;
  const size_t per_set = entry_a + entry_dt + 2 * entry_bc + entry_st;
  const size_t q = large ? k : std::max(k, std::min<size_t>((size_t)a->batch, ((size_t)16 << 20) / per_set));
  pl.set_entries = (int)q;
  pl.a_bytes = align_up(q * entry_a, 256);
  pl.dt_bytes = align_up(q * entry_dt, 256);
  pl.bc_bytes = align_up(q * entry_bc, 256);
  pl.enter_bytes = align_up(q * entry_st, 256);
  pl.st_bytes = align_up(k * entry_st, 256);
  // scratch of the forward: the largest need over every (entries, tokens) shape the pipeline will launch
  const std::vector<Slice> slices = make_slices(a, pl.tokens, pl.group, pl.set_entries);
  pl.nslices = (int)slices.size();
  pl.ws_bytes = 0;
  int seen_nb = -1, seen_tokens = -1;
  for (const Slice& sl : slices) {
    if (sl.nb == seen_nb && sl.tokens == seen_tokens) continue;
    seen_nb = sl.nb; seen_tokens = sl.tokens;
    SsdArgs s;
    chunk_args(a, sl.tokens, sl.nb, &s);
    pl.ws_bytes = std::max(pl.ws_bytes, align_up(ssd_b200_workspace_bytes(&s), 256));
  }
  // per-slice log-decay sums stay on the device until the end (one copy back)
  pl.ldall_bytes = a->final_logdecay ? align_up((size_t)pl.nslices * k * a->nheads * 4, 256) : 0;
  pl.slot_bytes = 2 * pl.x_bytes + pl.ws_bytes;
  // B, C, A, dt and the entering states travel per set, double-buffered
  pl.set_bytes = 2 * pl.bc_bytes + pl.a_bytes + pl.dt_bytes + pl.enter_bytes;
  // + the carried state (ping-pong) and the leaving state of a batch entry (two)
  // + every slice's log-decay sums + the status word of the kernels
  pl.total_bytes = kSlots * pl.slot_bytes + 2 * pl.set_bytes + 4 * pl.st_bytes + pl.ldall_bytes + 256;
  return pl;
}

}  // namespace

extern "C" {

size_t ssd_b200_host_scratch_bytes(const SsdArgs* host) {
  if (!basic_ok(host)) return 0;
  return make_plan(host).total_bytes;
}

int ssd_b200_forward_host(const SsdArgs* host, void* dev_scratch, size_t dev_scratch_bytes) {
  if (!host) return SSD_ERR_NULL_POINTER;
  if (!basic_ok(host)) {
    if (host->nheads > 0 && host->ngroups > 0 && host->chunk > 0 && host->seqlen > 0 &&
        host->nheads % host->ngroups == 0 && host->seqlen % host->chunk != 0)
      return SSD_ERR_BAD_CHUNK;
    return SSD_ERR_BAD_SHAPE;
  }
  const bool state_only = (host->flags & SSD_FLAG_STATE_ONLY) != 0;
  if (!host->X || !host->A || !host->B) return SSD_ERR_NULL_POINTER;
  if (!state_only && (!host->Y || !host->C)) return SSD_ERR_NULL_POINTER;
  if (state_only && !host->final_state) return SSD_ERR_NULL_POINTER;
  if (host->D || host->Z) return SSD_ERR_UNSUPPORTED;   // the skip/gate epilogue is a device-buffer feature
  const Plan pl = make_plan(host);
  if (!dev_scratch || dev_scratch_bytes < pl.total_bytes) return SSD_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(dev_scratch) & 255) return SSD_ERR_MISALIGNED;

  const int e = esize(host->dtype);
  const int b = host->batch, s = host->seqlen, h = host->nheads, p = host->headdim, n = host->dstate, g = host->ngroups;
  const std::vector<Slice> slices = make_slices(host, pl.tokens, pl.group, pl.set_entries);
  const int nslices = (int)slices.size();
  // The buffers of a set (B, C, A, dt, entering state) exist twice, and so does the leaving state of an entry (group).
  int last_run_user[2] = {-1, -1};     // last slice whose kernels read buffer set 0 / 1
  int last_leave_user[2] = {-1, -1};   // last slice whose final-state copy read the leaving-state buffer 0 / 1
  int nentries = 0, nsets = 0;
  const size_t np = (size_t)n * p;

  int rc = SSD_OK;
  auto ck = [&](cudaError_t err) { if (err != cudaSuccess && rc == SSD_OK) rc = SSD_ERR_CUDA; };
  // The three streams and the events of the pipeline are kept per device between calls (creating and destroying some
  // sixty events and three streams costs a few per cent of a 9 ms call); calls on one device take turns.
  int dev = 0;
  ck(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return SSD_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_pipes_mu[dev]);
  Pipe& pipe = g_pipes[dev];
  if (!pipe.st_in) ck(cudaStreamCreateWithFlags(&pipe.st_in, cudaStreamNonBlocking));
  if (!pipe.st_run) ck(cudaStreamCreateWithFlags(&pipe.st_run, cudaStreamNonBlocking));
  if (!pipe.st_out) ck(cudaStreamCreateWithFlags(&pipe.st_out, cudaStreamNonBlocking));
  while (rc == SSD_OK && (int)pipe.events.size() < 3 * nslices) {
    cudaEvent_t ev = nullptr;
    ck(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    if (ev) pipe.events.push_back(ev);
  }
  if (rc != SSD_OK) return rc;
  cudaStream_t st_in = pipe.st_in, st_run = pipe.st_run, st_out = pipe.st_out;
  cudaEvent_t* ev_in = pipe.events.data();
  cudaEvent_t* ev_run = ev_in + nslices;
  cudaEvent_t* ev_out = ev_run + nslices;

  char* base = static_cast<char*>(dev_scratch);
  char* set_base = base + kSlots * pl.slot_bytes;
  char* st_base = set_base + 2 * pl.set_bytes;
  float* carry[2] = {reinterpret_cast<float*>(st_base), reinterpret_cast<float*>(st_base + pl.st_bytes)};
  float* leave[2] = {reinterpret_cast<float*>(st_base + 2 * pl.st_bytes), reinterpret_cast<float*>(st_base + 3 * pl.st_bytes)};
  float* ld_all = reinterpret_cast<float*>(st_base + 4 * pl.st_bytes);   // [slice][entry of the group][head]
  int32_t* dev_status = reinterpret_cast<int32_t*>(st_base + 4 * pl.st_bytes + pl.ldall_bytes);
  // every kernel of the pipeline reports a wait that ran out to this word (the kernels run on st_run, in order)
  ck(cudaMemsetAsync(dev_status, 0, sizeof(int32_t), st_run));
  const char* hX = static_cast<const char*>(host->X);
  const char* hB = static_cast<const char*>(host->B);
  const char* hC = static_cast<const char*>(host->C);
  const char* hD = static_cast<const char*>(host->dt);
  char* hY = static_cast<char*>(host->Y);
  const bool want_state = host->final_state != nullptr;

  for (int i = 0; i < nslices && rc == SSD_OK; ++i) {
    const int bi = slices[i].bi, nb = slices[i].nb, ci = slices[i].ci, t0 = slices[i].t0, tokens = slices[i].tokens;
    const bool first = slices[i].first, last = slices[i].last;
    if (first) ++nentries;
    const int set = slices[i].set & 1, out = (nentries - 1) & 1;
    char* slot = base + (size_t)(i % kSlots) * pl.slot_bytes;
    char* dX = slot;
    char* dY = dX + pl.x_bytes;
    char* dW = dY + pl.x_bytes;
    float* dL = ld_all + (size_t)i * pl.group * h;
    char* eB = set_base + (size_t)set * pl.set_bytes;   // whole batch entries of the set: B, C, A, dt, entering state
    char* eC = eB + pl.bc_bytes;
    char* eA = eC + pl.bc_bytes;
    char* eD = eA + pl.a_bytes;
    float* enter = reinterpret_cast<float*>(eD + pl.dt_bytes);
    const size_t row = (size_t)(bi - slices[i].set_bi) * s + t0;   // first token of the chunk within the set
    char* dB = eB + row * g * n * e;
    char* dC = eC + row * g * n * e;
    char* dA = eA + row * h * 4;
    char* dD = eD + row * h * e;
    const size_t tok0 = (size_t)bi * s + t0;   // first token of the chunk in the [b*s] token axis

    // stage 1: copies in (the slot is free once the chunk that used it has left); every block is contiguous
    if (i >= kSlots) ck(cudaStreamWaitEvent(st_in, ev_out[i - kSlots], 0));
    if (slices[i].set == nsets) {
      // a new set; its buffers were last read by the kernels of the set before the last
      ++nsets;
      if (last_run_user[set] >= 0) ck(cudaStreamWaitEvent(st_in, ev_run[last_run_user[set]], 0));
      const size_t bi0 = (size_t)slices[i].set_bi, nb0 = (size_t)slices[i].set_nb, row0 = bi0 * s, rows = nb0 * s;
      ck(cudaMemcpyAsync(eB, hB + row0 * g * n * e, rows * g * n * e, cudaMemcpyHostToDevice, st_in));
      if (hC) ck(cudaMemcpyAsync(eC, hC + row0 * g * n * e, rows * g * n * e, cudaMemcpyHostToDevice, st_in));
      ck(cudaMemcpyAsync(eA, host->A + row0 * h, rows * h * 4, cudaMemcpyHostToDevice, st_in));
      if (hD) ck(cudaMemcpyAsync(eD, hD + row0 * h * e, rows * h * e, cudaMemcpyHostToDevice, st_in));
      if (host->initial_state)
        ck(cudaMemcpyAsync(enter, host->initial_state + bi0 * h * np, nb0 * h * np * 4, cudaMemcpyHostToDevice, st_in));
    }
    ck(cudaMemcpyAsync(dX, hX + tok0 * h * p * e, (size_t)nb * tokens * h * p * e, cudaMemcpyHostToDevice, st_in));
    last_run_user[set] = i;
    ck(cudaEventRecord(ev_in[i], st_in));

    // stage 2: kernels; the state enters from the previous chunk of the sequence and leaves for the next one
    ck(cudaStreamWaitEvent(st_run, ev_in[i], 0));
    if (last && want_state && last_leave_user[out] >= 0)
      ck(cudaStreamWaitEvent(st_run, ev_out[last_leave_user[out]], 0));
    SsdArgs sa;
    chunk_args(host, tokens, nb, &sa);
    sa.X = dX; sa.A = reinterpret_cast<const float*>(dA); sa.B = dB;
    sa.C = hC ? dC : nullptr;
    sa.dt = hD ? dD : nullptr;
    sa.Y = state_only ? nullptr : dY;
    sa.initial_state = first ? (host->initial_state ? enter + (size_t)(bi - slices[i].set_bi) * h * np : nullptr) : carry[(ci - 1) & 1];
    sa.final_state = last ? (want_state ? leave[out] : nullptr) : carry[ci & 1];
    sa.final_logdecay = host->final_logdecay ? dL : nullptr;
    sa.workspace = pl.ws_bytes ? dW : nullptr;
    sa.workspace_bytes = pl.ws_bytes;
    sa.status = dev_status;
    if (state_only && !sa.final_state) sa.final_state = carry[ci & 1];
    if (rc == SSD_OK) {
      const int frc = ssd_b200_forward(&sa, st_run);
      if (frc != SSD_OK) rc = frc;
    }
    ck(cudaEventRecord(ev_run[i], st_run));

    // stage 3: copies out
    ck(cudaStreamWaitEvent(st_out, ev_run[i], 0));
    if (!state_only)
      ck(cudaMemcpyAsync(hY + tok0 * h * p * e, dY, (size_t)nb * tokens * h * p * e, cudaMemcpyDeviceToHost, st_out));
    if (last && want_state) {
      ck(cudaMemcpyAsync(host->final_state + (size_t)bi * h * np, leave[out], (size_t)nb * h * np * 4,
                         cudaMemcpyDeviceToHost, st_out));
      last_leave_user[out] = i;
    }
    ck(cudaEventRecord(ev_out[i], st_out));
  }

  if (st_in) ck(cudaStreamSynchronize(st_in));
  if (st_run) ck(cudaStreamSynchronize(st_run));
  if (st_out) ck(cudaStreamSynchronize(st_out));
  int32_t dev_word = 0;
  if (rc == SSD_OK) ck(cudaMemcpy(&dev_word, dev_status, sizeof(dev_word), cudaMemcpyDeviceToHost));
  if (host->status) *host->status = dev_word;
  if (rc == SSD_OK && dev_word != 0) rc = SSD_ERR_DEVICE_WAIT;
  if (host->final_logdecay && rc == SSD_OK) {
    // per-slice sums, added up on the host
    std::vector<float> ld_host((size_t)nslices * pl.group * h, 0.f);
    ck(cudaMemcpy(ld_host.data(), ld_all, ld_host.size() * sizeof(float), cudaMemcpyDeviceToHost));
    std::vector<double> acc((size_t)b * h, 0.0);
    for (int i = 0; i < nslices; ++i)
      for (int eb = 0; eb < slices[i].nb; ++eb)
        for (int hh = 0; hh < h; ++hh)
          acc[(size_t)(slices[i].bi + eb) * h + hh] += ld_host[((size_t)i * pl.group + eb) * h + hh];
    for (size_t k = 0; k < acc.size(); ++k) host->final_logdecay[k] = (float)acc[k];
  }
  return rc;
}

}  // extern "C"
