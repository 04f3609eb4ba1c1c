#include "local_comm.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "../core/host_exec.h"
#include "../kernels/sar_params.h"
#include "../kernels/sar_cuda.h"
#include "symm_alloc.h"

namespace {
struct DevTable { SarOp* ops = nullptr; uint16_t* round_begin = nullptr; uint32_t num_rounds = 0, num_ops = 0; };
struct Rank {
  int dev = 0;
  cudaStream_t stream = nullptr;
  uint32_t* flags = nullptr;   // SAR_NUM_CHANNELS * SAR_FLAG_CAPACITY
  SarCtrl* ctrl = nullptr;     // SAR_NUM_CHANNELS
  uint32_t* status = nullptr;  // 1 word
  uint64_t* trace = nullptr;   // SAR_TRACE_WORDS words
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaEvent_t ev_in = nullptr;   // what the caller had queued (sar_local_wait_stream)
  bool timed = false;
  std::map<std::pair<uint64_t, int>, DevTable> tables;   // keyed by the table's contents, not its address
};
}  // namespace

struct sar_local_comm {
  int n = 0;
  bool emulate = false;
  std::vector<Rank> ranks;
  uint64_t epoch[SAR_NUM_CHANNELS] = {};   // 64-bit: the low word is the flag epoch, the whole value the gate base
  // emulate: blocks that fit the device, by (dtype, path, threads, ring stages, ops in the table)
  std::map<std::tuple<int, int, int, int, int>, int> resident;
  std::vector<sar::SymmAlloc*> allocs;   // symmetric buffers handed out by sar_local_alloc
};

// The symmetric allocation that holds bufs[r] for every rank at one common offset, or nullptr.
static const sar::SymmAlloc* find_alloc(const sar_local_comm* c, void* const* bufs, size_t bytes, size_t* offset) {
  for (const sar::SymmAlloc* a : c->allocs) {
    const char* b0 = (const char*)a->uc[0];
    const char* p0 = (const char*)bufs[0];
    if (p0 < b0 || p0 + bytes > b0 + a->mapped) continue;
    const size_t off = (size_t)(p0 - b0);
    bool same = true;
    for (int r = 1; r < c->n && same; ++r) same = (const char*)bufs[r] == (const char*)a->uc[r] + off;
    if (!same) continue;
    *offset = off;
    return a;
  }
  return nullptr;
}

#define CK(x)                                                                          \
  do {                                                                                 \
    cudaError_t e_ = (x);                                                              \
    if (e_ != cudaSuccess) {                                                           \
      if (err && errlen > 0) snprintf(err, errlen, "%s: %s", #x, cudaGetErrorString(e_)); \
      return fail_value;                                                               \
    }                                                                                  \
  } while (0)

// Content hash, eight bytes a step (a table is hashed for every rank of every call: byte by byte that was 13 us for
// the eight tables of `stragglar`, now under 2).  The shift brings the high bytes of a word into the low bits.
static uint64_t hash_bytes(uint64_t h, const void* p, size_t n) {
  const unsigned char* c = (const unsigned char*)p;
  for (; n >= 8; c += 8, n -= 8) {
    uint64_t v;
    memcpy(&v, c, 8);
    h = (h ^ v) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 29;
  }
  for (; n; ++c, --n) h = (h ^ *c) * 0x100000001b3ull;
  return h;
}

// Device copy of a rank's table.  The cache is keyed by a hash of the table's
// contents: programs come and go on the host, and a new one may live at the
// address of one that was freed.
static DevTable* upload(Rank& rk, const sar_table* t, int rank, char* err, int errlen) {
  const int nops = sar_table_num_ops(t, rank);
  const int nrb = sar_table_num_round_begin(t, rank);
  uint64_t h = 0xcbf29ce484222325ull;
  if (nops) h = hash_bytes(h, sar_table_ops(t, rank), sizeof(SarOp) * nops);
  if (nrb) h = hash_bytes(h, sar_table_round_begin(t, rank), sizeof(uint16_t) * nrb);
  h = hash_bytes(h, &nops, sizeof nops);
  auto key = std::make_pair(h, rank);
  auto it = rk.tables.find(key);
  if (it != rk.tables.end()) return &it->second;
  DevTable* fail_value = nullptr;
  {
    char why[200] = "";
    if (sar_table_validate(t, rank, sar_table_nranks(t), why, sizeof why)) {
      if (err && errlen > 0) snprintf(err, errlen, "refusing to launch a malformed table (%s): %s", sar_status_string(SAR_BAD_TABLE), why);
      return nullptr;
    }
  }
  DevTable d;
  CK(cudaMalloc(&d.ops, sizeof(SarOp) * (nops > 0 ? nops : 1)));
  CK(cudaMalloc(&d.round_begin, sizeof(uint16_t) * (nrb > 0 ? nrb : 1)));
  if (nops) CK(cudaMemcpy(d.ops, sar_table_ops(t, rank), sizeof(SarOp) * nops, cudaMemcpyHostToDevice));
  if (nrb) CK(cudaMemcpy(d.round_begin, sar_table_round_begin(t, rank), sizeof(uint16_t) * nrb, cudaMemcpyHostToDevice));
  d.num_rounds = nrb > 0 ? (uint32_t)(nrb - 1) : 0;
  d.num_ops = nops > 0 ? (uint32_t)nops : 0;
  return &(rk.tables[key] = d);
}

// Launch shape of a collective whose ranks share one device: as many blocks per rank as can be resident together,
// but no more than one per 16 KiB of a rank's buffer (tiles start at 2 KiB: below that the blocks find no work and
// only lengthen the entry).  Every block is a serial chain of wait, move, announce, so bandwidth comes from their
// number.  On the simt paths 256 threads a block let three chains share an SM where 512 leave it one (sar_emul_simt_kernel),
// on the bulk-copy path three ring stages two (tma::Shared).  8 ranks, fp32, against 4 blocks per rank: 25 MiB 123 us
// against 563, 256 MiB 0.97 ms against 5.41; 6 ranks, simt, 12 MB 64 us against 230.
// The launch is cooperative, so it starts when the whole device is free for it.
static int emulated_blocks(sar_local_comm* c, const sar_program* prog, int dtype, int path, int* threads, int stages, uint64_t bytes) {
  if (path == SAR_PATH_SIMTA || (path == SAR_PATH_SIMT && *threads <= 0)) *threads = 256;
  cudaSetDevice(c->ranks[0].dev);   // occupancy is that of the current device
  int nops = 0;
  if (path != SAR_PATH_SIMTA)
    for (int ph = 0; ph < sar_program_num_phases(prog); ++ph)
      for (int r = 0; r < c->n; ++r) nops = std::max(nops, sar_table_num_ops(sar_program_phase(prog, ph), r));
  const auto key = std::make_tuple(dtype, path, *threads, stages, nops);
  auto it = c->resident.find(key);
  if (it == c->resident.end()) it = c->resident.emplace(key, sar_cuda_emulated_fit(dtype, path, *threads, stages, nops)).first;
  const uint64_t fit = (uint64_t)(it->second / c->n), want = (bytes + (16u << 10) - 1) / (16u << 10);
  const uint64_t b = want < 4 ? 4 : want;
  return (int)(b < fit ? b : (fit < 1 ? 1 : fit));
}

extern "C" {

sar_local_comm* sar_local_create(int n, const int* devices, int emulate, char* err, int errlen) {
  sar_local_comm* fail_value = nullptr;
  if (n < 1 || n > SAR_MAX_RANKS) {
    if (err) snprintf(err, errlen, "rank count %d out of range", n);
    return nullptr;
  }
  auto* c = new sar_local_comm;
  c->n = n; c->emulate = emulate != 0;
  c->ranks.resize(n);
  for (int r = 0; r < n; ++r) {
    Rank& rk = c->ranks[r];
    rk.dev = emulate ? devices[0] : devices[r];
    CK(cudaSetDevice(rk.dev));
    if (emulate && r > 0) rk.stream = c->ranks[0].stream;
    else CK(cudaStreamCreateWithFlags(&rk.stream, cudaStreamNonBlocking));
    const size_t fbytes = sizeof(uint32_t) * SAR_NUM_CHANNELS * (size_t)SAR_FLAG_CAPACITY;
    CK(cudaMalloc(&rk.flags, fbytes));
    CK(cudaMemset(rk.flags, 0, fbytes));
    CK(cudaMalloc(&rk.ctrl, sizeof(SarCtrl) * SAR_NUM_CHANNELS));
    CK(cudaMemset(rk.ctrl, 0, sizeof(SarCtrl) * SAR_NUM_CHANNELS));
    CK(cudaMalloc(&rk.status, 16));
    CK(cudaMemset(rk.status, 0, 16));
    CK(cudaMalloc(&rk.trace, sizeof(uint64_t) * SAR_TRACE_WORDS));
    CK(cudaMemset(rk.trace, 0, sizeof(uint64_t) * SAR_TRACE_WORDS));
    CK(cudaEventCreate(&rk.ev0));
    CK(cudaEventCreate(&rk.ev1));
    CK(cudaEventCreateWithFlags(&rk.ev_in, cudaEventDisableTiming));
  }
  if (!emulate) {
    for (int a = 0; a < n; ++a) {
      CK(cudaSetDevice(c->ranks[a].dev));
      for (int b = 0; b < n; ++b) {
        if (a == b || c->ranks[a].dev == c->ranks[b].dev) continue;
        int can = 0;
        CK(cudaDeviceCanAccessPeer(&can, c->ranks[a].dev, c->ranks[b].dev));
        if (!can) {
          if (err) snprintf(err, errlen, "device %d cannot access device %d", c->ranks[a].dev, c->ranks[b].dev);
          return nullptr;
        }
        cudaError_t e = cudaDeviceEnablePeerAccess(c->ranks[b].dev, 0);
        if (e == cudaErrorPeerAccessAlreadyEnabled) cudaGetLastError();
        else CK(e);
      }
    }
  }
  for (int r = 0; r < n; ++r) { CK(cudaSetDevice(c->ranks[r].dev)); CK(cudaDeviceSynchronize()); }
  return c;
}

void sar_local_destroy(sar_local_comm* c) {
  if (!c) return;
  for (int r = 0; r < c->n; ++r) {
    Rank& rk = c->ranks[r];
    cudaSetDevice(rk.dev);
    cudaDeviceSynchronize();
    for (auto& kv : rk.tables) { cudaFree(kv.second.ops); cudaFree(kv.second.round_begin); }
    cudaFree(rk.flags); cudaFree(rk.ctrl); cudaFree(rk.status); cudaFree(rk.trace);
    cudaEventDestroy(rk.ev0); cudaEventDestroy(rk.ev1); cudaEventDestroy(rk.ev_in);
    if (!(c->emulate && r > 0)) cudaStreamDestroy(rk.stream);
  }
  for (sar::SymmAlloc* a : c->allocs) { sar::symm_free(a); delete a; }
  delete c;
}

int sar_local_nranks(const sar_local_comm* c) { return c->n; }
void* sar_local_stream(sar_local_comm* c, int rank) { return c->ranks[rank].stream; }

int sar_local_wait_stream(sar_local_comm* c, int rank, void* stream) {
  Rank& rk = c->ranks[rank];
  cudaError_t e = cudaSetDevice(rk.dev);
  if (e == cudaSuccess) e = cudaEventRecord(rk.ev_in, (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(rk.stream, rk.ev_in, 0);
  return (int)e;
}

int sar_local_run(sar_local_comm* c, const sar_program* prog, void* const* bufs, uint64_t count, int dtype,
                  const sar_run_opts* o, const uint64_t* delay_ns, char* err, int errlen) {
  int fail_value = 1;
  const int n = c->n;
  const int nph = sar_program_num_phases(prog);
  if (nph < 1 || sar_table_nranks(sar_program_phase(prog, 0)) != n) {
    if (err) snprintf(err, errlen, "program is for %d ranks, communicator has %d", nph ? sar_table_nranks(sar_program_phase(prog, 0)) : 0, n);
    return 1;
  }
  if (o->user_in && o->user_out && nph != 1) {
    if (err) snprintf(err, errlen, "staged mode serves single-phase programs");
    return 1;
  }
  for (int r = 0; r < n; ++r)
    if (((uintptr_t)bufs[r]) & 15) { if (err) snprintf(err, errlen, "buffer of rank %d is not 16-byte aligned", r); return 1; }
  const uint32_t esize = dtype == SAR_F32 ? 4 : 2;
  const int path = o->path;
  int blocks = o->blocks > 0 ? o->blocks : sar_cuda_pick_blocks(path, count * esize);
  int threads = path == SAR_PATH_SIMT ? o->threads : 0, stages = o->stages;
  if (c->emulate && o->blocks <= 0) {
    if (path == SAR_PATH_TMA && stages <= 0) stages = 3;   // two blocks per SM (see tma::Shared)
    blocks = emulated_blocks(c, prog, dtype, path, &threads, stages, count * esize);
  }
  const bool lone = n == 1 && !c->emulate && o->blocks <= 0;
  if (lone) { blocks = sar_cuda_lone_blocks(count * esize); if (stages <= 0) stages = 6; }
  const double timeout_s = o->timeout_s > 0 ? o->timeout_s : 10.0;
  // Emulated ranks, simt and simta: tiles of up to 256 KiB, because the wait, the block barriers and the fence around
  // a tile are not hidden behind another one (256 / 128 / 64 KiB: ring, 4 ranks, 40 MB 112 / 113 / 120 us, simta
  // 116 / 116 / 124 us; rhd, 8 ranks, 64 MiB fp16 386 / 386 / 402 us, simta 394 / 403 / 398 us; level where the blocks
  // outnumber the tiles).  The bulk-copy ring hides them: 64 KiB (8 ranks, 25 MiB 124 us against 129 with 32, 128 or
  // 256 KiB; 256 MiB 968 against 976, 977 and 1033 us with 128, 256 and 32 KiB).
  const uint32_t tile_max = o->tile_bytes ? o->tile_bytes : lone ? sar_cuda_lone_tile_bytes(path)
                          : (c->emulate && path != SAR_PATH_TMA ? (256u << 10) : sar_cuda_default_tile_bytes(path));
  std::vector<bool> delayed(n, false);

  for (int r = 0; r < n; ++r) c->ranks[r].timed = o->timed != 0;

  // multicast views of the buffers, when they come from sar_local_alloc (simt path only: multimem
  // instructions are issued by threads, not by the bulk-copy engine)
  size_t mc_off = 0;
  const sar::SymmAlloc* mc_alloc = nullptr;
  if (!c->emulate && path != SAR_PATH_TMA && !c->allocs.empty()) {
    mc_alloc = find_alloc(c, bufs, (size_t)count * esize, &mc_off);
    if (mc_alloc && !mc_alloc->mc_handle[0]) mc_alloc = nullptr;
  }

  // ---- prepare every phase: geometry, device tables (uploaded on first use), launch parameters
  struct PhaseLaunch { std::vector<SarLaunchParams> hp; int blocks; uint32_t parts; };
  std::vector<PhaseLaunch> launches(nph);
  for (int ph = 0; ph < nph; ++ph) {
    const sar_table* t = sar_program_phase(prog, ph);
    const int ch = sar_table_channel(t);
    const uint32_t parts = sar_table_participants(t);
    const uint32_t nch = (uint32_t)sar_table_num_chunks(t);
    c->epoch[ch] += SAR_VER_STRIDE;
    int pblocks = blocks;   // this phase's block count: the table may ask for fewer
    const int hint = sar_table_blocks_hint(t);
    if (o->blocks <= 0 && !c->emulate && hint > 0 && hint < pblocks) pblocks = hint;
    // Gating keeps the rounds of a matching-based schedule from contending for the ports of the switch.  Emulated
    // ranks have no ports, only the hand-shake's cost (256 MiB, 8 ranks: 1061 us gated, 964 us free-running): they
    // are gated when that was asked for (STRAGGLAR_GATE, read when the program is compiled).
    const bool gate_wanted = !c->emulate || sar_table_gate_asked(t);
    const bool gated = gate_wanted && sar_table_gate_rounds(t) && count * esize >= sar_gate_min_bytes();
    const uint32_t ptile_max = (gated && !o->tile_bytes && !c->emulate) ? sar::gate_tile_bytes() : tile_max;
    const uint32_t tile_elems = sar_pick_tile_elems(count, esize, nch, (uint32_t)pblocks, 2048, ptile_max);
    SarGeom g = sar::make_geom(count, esize, nch, tile_elems);
    if ((uint64_t)g.tiles_per_chunk * g.num_chunks > SAR_FLAG_CAPACITY) {
      if (err) snprintf(err, errlen, "buffer too large for the flag array");
      return 1;
    }
    PhaseLaunch& L = launches[ph];
    L.hp.resize(n); L.blocks = pblocks; L.parts = parts;
    for (int r = 0; r < n; ++r) {
      Rank& rk = c->ranks[r];
      SarLaunchParams& P = L.hp[r];
      memset(&P, 0, sizeof(P));
      for (int q = 0; q < n; ++q) {
        P.comm.flags[q] = c->ranks[q].flags + (size_t)ch * SAR_FLAG_CAPACITY;
        P.comm.ctrl[q] = c->ranks[q].ctrl + ch;
        P.comm.buf[q] = bufs[q];
      }
      CK(cudaSetDevice(rk.dev));
      DevTable* dt = upload(rk, t, r, err, errlen);
      if (!dt) return 1;
      P.ops = dt->ops; P.round_begin = dt->round_begin; P.num_rounds = dt->num_rounds; P.num_ops = dt->num_ops;
      P.one_device = c->emulate || n == 1;
      P.geom = g; P.rank = r; P.nranks = n; P.participants = parts;
      P.epoch_base = (uint32_t)c->epoch[ch]; P.gate_base = c->epoch[ch]; P.scale = o->scale; P.dtype = dtype;
      P.timeout_ns = (uint64_t)(timeout_s * 1e9);
      P.status = rk.status; P.trace = rk.trace; P.trace_rounds = o->trace_rounds ? 1u : 0u;
      P.gate_rounds = gated ? 1u : 0u;
      P.gate_slack = sar::gate_slack(g.tiles_per_chunk);
      P.stages = stages > 0 ? (uint32_t)stages : (uint32_t)sar_table_stages_hint(t);
      P.lane1_eighths = (uint32_t)sar_table_lane1_eighths(t);
      if (mc_alloc) {
        for (int grp = 0; grp < 2; ++grp) {
          if (!mc_alloc->mc[grp][r]) continue;
          P.mc[grp].base = (char*)mc_alloc->mc[grp][r] + mc_off;
          P.mc[grp].members = mc_alloc->members[grp];
        }
      }
      if (o->user_in && o->user_out) {
        P.user_in = o->user_in[r]; P.user_out = o->user_out[r]; P.user_dtype = o->user_dtype;
        sar_table_final_ver(t, r, P.final_ver);
        if ((c->emulate || n == 1) && o->blocks <= 0) P.staging_blocks = SAR_STAGE_EVERYWHERE;
      }
      P.delay_ns = 0;
      if (c->emulate && delay_ns && delay_ns[r] && !delayed[r] && (parts >> r & 1)) { P.delay_ns = delay_ns[r]; delayed[r] = true; }
    }
  }

  if (o->trace_rounds) {
    // start stamps begin at the maximum (they are lowered with atomicMin), the rest at zero
    for (int r = 0; r < n; ++r) {
      Rank& rk = c->ranks[r];
      CK(cudaSetDevice(rk.dev));
      CK(cudaMemsetAsync(rk.trace + 2, 0xff, sizeof(uint64_t) * SAR_MAX_ROUNDS, rk.stream));
      CK(cudaMemsetAsync(rk.trace + 2 + SAR_MAX_ROUNDS, 0, sizeof(uint64_t) * 2 * SAR_MAX_ROUNDS, rk.stream));
    }
  }

  if (c->emulate) {
    // every rank on one device: one cooperative launch per phase on one stream
    Rank& r0 = c->ranks[0];
    CK(cudaSetDevice(r0.dev));
    if (o->timed) CK(cudaEventRecord(r0.ev0, r0.stream));
    for (int ph = 0; ph < nph; ++ph) {
      cudaError_t e = (cudaError_t)sar_cuda_launch_emulated(launches[ph].hp.data(), n, path, launches[ph].blocks, threads, r0.stream);
      if (e != cudaSuccess) {
        if (err) snprintf(err, errlen, "emulated launch (%d ranks x %d blocks): %s", n, launches[ph].blocks, cudaGetErrorString(e));
        return (int)e;
      }
    }
    if (o->timed) CK(cudaEventRecord(r0.ev1, r0.stream));
    return 0;
  }

  // ---- one rank per device.  Everything of a rank is enqueued before the next rank is touched:
  // [start barrier, start event,] [delay,] its phases [, stop event].  The start barrier holds
  // every stream until the last rank's barrier kernel runs, by which time the work of all
  // other ranks is already queued behind theirs, so the host's launch order stays out of the
  // timed window.
  uint32_t barrier_epoch = 0;
  SarCtrl* bctrl[SAR_MAX_RANKS] = {};
  if (o->timed) {
    barrier_epoch = (uint32_t)++c->epoch[SAR_NUM_CHANNELS - 1];
    for (int r = 0; r < n; ++r) bctrl[r] = c->ranks[r].ctrl + (SAR_NUM_CHANNELS - 1);
  }
  for (int r = 0; r < n; ++r) {
    Rank& rk = c->ranks[r];
    CK(cudaSetDevice(rk.dev));
    if (o->timed) {
      CK((cudaError_t)sar_cuda_barrier(bctrl, r, n, (1u << n) - 1u, barrier_epoch, (uint64_t)(timeout_s * 1e9), rk.status, rk.stream));
      CK(cudaEventRecord(rk.ev0, rk.stream));
    }
    for (int ph = 0; ph < nph; ++ph) {
      if (!(launches[ph].parts >> r & 1)) continue;
      if (delay_ns && delay_ns[r] && !delayed[r]) { CK((cudaError_t)sar_cuda_delay(delay_ns[r], rk.stream)); delayed[r] = true; }
      CK((cudaError_t)sar_cuda_launch(&launches[ph].hp[r], path, launches[ph].blocks, threads, rk.stream));
    }
    if (o->timed) CK(cudaEventRecord(rk.ev1, rk.stream));
  }
  return 0;
}

int sar_local_round_trace(sar_local_comm* c, uint64_t* out) {
  for (int r = 0; r < c->n; ++r) {
    cudaSetDevice(c->ranks[r].dev);
    cudaError_t e = cudaMemcpy(out + (size_t)r * 3 * SAR_MAX_ROUNDS, c->ranks[r].trace + 2, sizeof(uint64_t) * 3 * SAR_MAX_ROUNDS,
                               cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

int sar_local_alloc(sar_local_comm* c, size_t bytes, int mode, uint32_t sub_members, void** bufs, char* err, int errlen) {
  int devs[SAR_MAX_RANKS];
  for (int r = 0; r < c->n; ++r) devs[r] = c->ranks[r].dev;
  if (c->emulate) {
    if (mode == sar::SYMM_MULTICAST) {
      if (err) snprintf(err, errlen, "multicast needs one device per rank (the ranks are emulated on one device)");
      return 1;
    }
    mode = sar::SYMM_PLAIN;
  }
  auto* a = new sar::SymmAlloc;
  if (sar::symm_alloc(a, c->n, devs, bytes, mode, sub_members, err, errlen) != 0) { delete a; return 1; }
  for (int r = 0; r < c->n; ++r) bufs[r] = a->uc[r];
  c->allocs.push_back(a);
  return 0;
}

int sar_local_free(sar_local_comm* c, void* buf0) {
  for (size_t i = 0; i < c->allocs.size(); ++i) {
    if (c->allocs[i]->uc[0] != buf0) continue;
    sar::symm_free(c->allocs[i]);
    delete c->allocs[i];
    c->allocs.erase(c->allocs.begin() + (long)i);
    return 0;
  }
  return 1;
}

int sar_local_multicast_groups(sar_local_comm* c, const void* buf0) {
  for (const sar::SymmAlloc* a : c->allocs) {
    const char* b0 = (const char*)a->uc[0];
    if ((const char*)buf0 < b0 || (const char*)buf0 >= b0 + a->mapped) continue;
    return (a->mc_handle[0] ? 1 : 0) | (a->mc_handle[1] ? 2 : 0);
  }
  return 0;
}

int sar_local_multicast_supported(sar_local_comm* c) {
  if (c->emulate) return 0;
  int devs[SAR_MAX_RANKS];
  for (int r = 0; r < c->n; ++r) {
    devs[r] = c->ranks[r].dev;
    for (int q = 0; q < r; ++q) if (devs[q] == devs[r]) return 0;
  }
  return sar::multicast_supported(c->n, devs) ? 1 : 0;
}

uint32_t sar_local_sync(sar_local_comm* c, float* ms) {
  uint32_t worst = 0;
  for (int r = 0; r < c->n; ++r) {
    Rank& rk = c->ranks[r];
    cudaSetDevice(rk.dev);
    cudaError_t e = cudaStreamSynchronize(rk.stream);
    if (e != cudaSuccess) { worst = 0x1000u + (uint32_t)e; continue; }
    uint32_t st = 0;
    cudaMemcpy(&st, rk.status, 4, cudaMemcpyDeviceToHost);
    if (st) {
      worst = worst > st ? worst : st;
      cudaMemset(rk.status, 0, 4);
      for (int ch = 0; ch < SAR_NUM_CHANNELS; ++ch) {
        cudaMemset(&rk.ctrl[ch].abort_flag, 0, 4);
        cudaMemset(&rk.ctrl[ch].blocks_done, 0, 4);
      }
    }
    if (ms) {
      ms[r] = 0.f;
      const Rank& ev = c->emulate ? c->ranks[0] : rk;
      if (rk.timed) cudaEventElapsedTime(&ms[r], ev.ev0, ev.ev1);
    }
  }
  return worst;
}

int sar_local_trace(sar_local_comm* c, uint64_t* out) {
  for (int r = 0; r < c->n; ++r) {
    cudaSetDevice(c->ranks[r].dev);
    cudaError_t e = cudaMemcpy(out + 2 * r, c->ranks[r].trace, 16, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}
}
