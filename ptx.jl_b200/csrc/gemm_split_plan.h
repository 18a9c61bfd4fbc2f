// Sizes of gemm_split_sm100.cu that the kernel, its launcher and the CPU tests share: ring
// stages, chains of partial sums, shared and tensor memory of a CTA. Plain C++.
#pragma once

#if defined(__CUDACC__)
#define PTXB200_PLAN_HD __host__ __device__
#else
#define PTXB200_PLAN_HD
#endif

namespace ptxb200 {

constexpr int kBM3 = 128;             // rows of a tile
constexpr int kBK3 = 64;              // a step of K: one 128-byte swizzle row of bf16
constexpr int kMaxStages3 = 7;
constexpr int kSmemMax3 = 232448;     // what a CTA can opt in to
constexpr int kABytes3 = kBM3 * kBK3 * 2;
constexpr int kChainSteps3 = 8;       // steps of K per accumulator
// full[], empty[], acc_full[2], acc_empty[2], parts_in, TMEM slot, abort flag
constexpr int kCtrlBytes3 = ((2 * kMaxStages3 + 5) * 8 + 8 + 15) / 16 * 16;
static_assert(kCtrlBytes3 % 16 == 0, "the parts handed over behind it are 16-byte pieces");

// steps of K per ring stage: two of 24 KiB (64 columns), or one of 32 or 40 KiB
PTXB200_PLAN_HD constexpr int stage_k3(int bn) { return bn == 64 ? 2 : 1; }
PTXB200_PLAN_HD constexpr int stage_bytes3(int bn) { return stage_k3(bn) * (kABytes3 + bn * kBK3 * 2); }
// accumulators that tensor memory (512 columns) holds; with more chains of sums than that, two
// take turns and a third block of columns keeps what has been added up
PTXB200_PLAN_HD constexpr int max_accs3(int bn) { return 512 / bn; }
// columns [part_col3(.., part), part_col3(.., part + 1)) of a tile are added up by one of its CTAs;
// the kernel has the first columns of all parts in one word, four bits each, in units of 16 (a
// division there costs 0.1 us behind the last product)
constexpr int part_col3(int bn, int split, int part) { return bn / 16 * part / split * 16; }
inline unsigned long long part_cols3(int bn, int split) {
  unsigned long long word = 0;
  for (int part = 0; part <= split; ++part) word |= (unsigned long long)(part_col3(bn, split, part) / 16) << (4 * part);
  return word;
}
PTXB200_PLAN_HD constexpr int unpack_col3(unsigned long long word, int part) { return (int)(word >> (4 * part) & 15) * 16; }
// what the other parts of the tile hand a CTA: [split - 1][columns / 4][128 rows] float4; a slot
// has room for the widest share
constexpr int slot_bytes3(int bn, int split) { return kBM3 * ((bn / 16 + split - 1) / split * 16) * 4; }
constexpr int recv_bytes3(int bn, int split) { return (split - 1) * slot_bytes3(bn, split); }
// steps [part_begin3(.., part), part_begin3(.., part + 1)) of K are one CTA's
PTXB200_PLAN_HD constexpr int part_begin3(int kiters, int split, int part) {
  return (int)((unsigned)kiters * (unsigned)part / (unsigned)split);   // K < 2^31: the product fits
}

constexpr int kMaxParts3 = 8;
constexpr int kLongSteps3 = 192;      // steps of K from which handing over up to 7 shares pays
struct GemmSplitPlan {
  int bn;         // columns of a tile (128 rows): 64, 128 or 192
  int split;      // parts of K, one CTA of a cluster each: 1 to 8
};

// Which products run on small tiles, and how: those whose 128x128 tiles fit the SMs in one round
// (more tiles are better off in the persistent kernels: 2048x2048x512 9.1 us there, 9.1-11.2 here).
// Tiles of 64 columns if those fit too, since a step of K costs a CTA nearly the same for
// 64 columns as for 128 (1024^3: 6.7 against 7.7 us). K is split where SMs are left over and a
// part keeps at least 4 (split in 4) or 8 (in 2) steps: handing the parts over costs
// 1-2 us (384x640x1024: 5.8 in 4 parts, 6.7 whole; 512^3: 5.4 in 2 or 4 parts, 4.9 whole).
// In 4 only where all clusters run at once (`clusters[4]`): 34 products of 128x64x1024 take two
// rounds and 11.8 us in 4 parts, 8.0 in 2; 33 take 7.8 and 8.0.
// Half of K on tiles of 128 columns against all of it on tiles of 64, which use equally
// many CTAs, pays from about 64 steps on (1024x1152: 16.1 against 16.5 us at 64 steps, 21.0
// against 25.3 at 128, 11.7 against 10.5 at 32).
// Long K: 128 columns in as many parts as run at once, down to 3 (but 8 or none where 64 columns
// go in 4: 512x512x32768 34.1 us in 6 parts of 128 columns, 30.7 in 4 of 64), and 192 columns in 2
// where a whole K on 128 leaves up to half of the SMs idle. 512x640x32768 47.7 -> 35.0 us,
// 256x512x65536 49.0 -> 40.3, 640x1024x16384 33 (shares of one line of steps over all SMs) -> 29.3,
// 1024x1280x16384 57.2 -> 49.0. The lines cross between 64 and 192 steps: at 128, 640x1024 21.2
// and 18.6 but 128x10240 38.6 and 40.4; from 192 on none of 24 shapes was slower by more than 2 %.
inline bool gemm_split_rule(int sm_count, const int* clusters, int groups, int M, int N, int kiters, bool may_split,
                            GemmSplitPlan* plan) {
  const long long sms = sm_count, rows = (long long)groups * (M / kBM3);
  const long long tiles128 = rows * ((N + 127) / 128), tiles64 = rows * ((N + 63) / 64);
  if (tiles128 > sms) return false;
  if (may_split && kiters >= kLongSteps3) {
    const int parts[] = {8, 6, 5, 4, 3};
    for (int s : parts)
      if (tiles128 <= clusters[s] && (s == 8 || tiles64 > clusters[4])) {
        plan->bn = 128;
        plan->split = s;
        return true;
      }
    if (tiles128 * 2 > sms && rows * ((N + 191) / 192) * 2 <= sms) {
      plan->bn = 192;
      plan->split = 2;
      return true;
    }
  }
  plan->split = 1;
  if (tiles64 > sms || (may_split && kiters >= 64 && tiles64 * 2 > sms && tiles128 * 2 <= sms)) {
    plan->bn = 128;
    if (may_split && kiters >= 16 && tiles128 * 2 <= sms) plan->split = 2;
    return true;
  }
  plan->bn = 64;
  if (may_split && kiters >= 16) plan->split = tiles64 <= clusters[4] ? 4 : tiles64 * 2 <= sms ? 2 : 1;
  return true;
}

// Few 128x256 tiles, cut along K: the steps of all tiles as one line, dealt out in equal shares of
// at least kLineMinSteps to at most one CTA per SM, where that gives every tile two CTAs or more.
constexpr int kLineMinSteps = 8;
struct GemmLine {
  int ctas;       // 0: not cut
  int share;      // steps of the longest share, or all of K
};
inline GemmLine gemm_line(int sm_count, int groups, int M, int N, int kiters) {
  const long long tiles = (long long)groups * (M / kBM3) * ((N + 255) / 256), line = tiles * kiters;
  long long ctas = line / kLineMinSteps;
  if (ctas > sm_count) ctas = sm_count;
  if (tiles * 2 > sm_count || ctas < 2 * tiles) return {0, kiters};
  return {(int)ctas, (int)((line + ctas - 1) / ctas)};
}

struct GemmSplitLayout {
  int stages;         // of the ring
  int chain_stages;   // stages a chain of sums runs over
  bool fold;          // K split, more chains than accumulators (in the longest part; the same for all)
  int tmem_cols;
  int smem_bytes;
};

// `longest`: steps that no chain of sums may exceed (but kChainSteps3), 0: one chain over all of a
// part's K. fp32 output has chains of kChainSteps3 steps, longer ones only where that saves folding.
inline GemmSplitLayout gemm_split_layout(const GemmSplitPlan& p, int kiters, bool f32, int longest) {
  GemmSplitLayout l;
  // a ring as deep as shared memory allows, but no deeper than the work
  const int recv = recv_bytes3(p.bn, p.split), per = stage_k3(p.bn);
  const int steps = ((kiters + p.split - 1) / p.split + per - 1) / per;   // of the longest part, in stages
  l.stages = (kSmemMax3 - kCtrlBytes3 - recv) / stage_bytes3(p.bn);
  if (l.stages > kMaxStages3) l.stages = kMaxStages3;
  if (l.stages > steps) l.stages = steps;
  const int shortest = kChainSteps3 / per, limit = longest / per > shortest ? longest / per : shortest;   // stages
  l.chain_stages = longest == 0 || steps <= shortest ? steps : f32 ? shortest : limit;
  int chains = (steps + l.chain_stages - 1) / l.chain_stages;
  const int accs = max_accs3(p.bn);
  if (p.split > 1 && chains > accs && (steps + accs - 1) / accs <= limit) chains = accs;
  l.fold = p.split > 1 && chains > accs;
  l.chain_stages = (steps + chains - 1) / chains;
  l.tmem_cols = 64;      // a power of two
  const int blocks = l.fold ? 3 : p.split > 1 || chains < 2 ? chains : 2;
  while (l.tmem_cols < blocks * p.bn) l.tmem_cols *= 2;
  l.smem_bytes = l.stages * stage_bytes3(p.bn) + kCtrlBytes3 + recv;
  // Two CTAs of different clusters never share an SM: each could hold the tensor memory that the
  // other's peers wait for. (An SM has 1 KiB more than a CTA can take, and a CTA costs it 1 KiB.)
  if (p.split > 1 && l.smem_bytes <= kSmemMax3 / 2) l.smem_bytes = kSmemMax3 / 2 + 16;
  return l;
}

}  // namespace ptxb200
