// rk_conf.cuh -- the Particles and Interactions sections of a conf file,
// formatted on the device (Rockable::saveConf, Rockable.cpp:547-580), for
// rk_format_conf in rk_api.cu.  A warp writes the line of a body or an active
// entry into a fixed-size slot (rk_fmt.cuh's exact printf("%.*e")), the line
// lengths are prefix-summed, and the lines are packed into one text.
#pragma once
#include "rk_engine.cuh"
#include "rk_fmt.cuh"

namespace rk {

constexpr int kConfBodySlot = 1024;  // name (<= 255) + 2 integers + 20 numbers of <= 26 characters
constexpr int kConfEntrySlot = 512;  // 5 integers + 17 numbers
constexpr int kConfMaxName = 255;

// The fields of one line, a lane each (text of len characters in cell): put
// one after the other in o, separated by spaces, closed by a newline; returns
// the line's length.  One thread per line formatted its 17 to 20 numbers one
// after the other, on few warps: 20 000 bodies and 49 000 contacts took 0.35
// and 1.61 ms.
constexpr int kConfCell = 32;  // a number or an integer has at most 26 characters
__device__ __forceinline__ int conf_line(const char* cell, int len, int fields, char* o) {
  const int lane = threadIdx.x & 31;
  const int width = lane < fields ? len + 1 : 0;  // with the space or the newline behind it
  int end = width;
  for (int q = 1; q < 32; q <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, end, q);
    if (lane >= q) end += y;
  }
  if (lane < fields) {
    char* at = o + end - width;
    if (cell)
      for (int k = 0; k < len; k++) at[k] = cell[k];
    at[len] = lane == fields - 1 ? '\n' : ' ';
  }
  return __shfl_sync(0xffffffffu, end, 31);
}

// "name group cluster homothety pos vel acc Q vrot arot\n", one warp per body
__global__ void k_conf_bodies(Scene s, const char* names, const int* name_ofs, int prec, char* slots,
                              int64_t* lens) {
  const int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (b >= s.n) return;
  char* o = slots + b * (int64_t)kConfBodySlot;
  const int sh = s.shape[b];
  const int n0 = name_ofs[sh];
  int nl = name_ofs[sh + 1] - n0;
  if (nl > kConfMaxName) nl = kConfMaxName;
  for (int k = lane; k < nl; k += 32) o[k] = names[n0 + k];
  char cell[kConfCell];
  int len = 0;
  if (lane == 0) len = nl;  // (the name is in place)
  else if (lane == 1) len = fmt_i(s.group[b], cell);
  else if (lane == 2) len = fmt_i(s.cluster[b], cell);
  else if (lane < 23) {
    double x;
    const int f = lane - 4;  // 19 numbers behind the homothety
    if (f < 0) x = s.hom[b];
    else if (f < 9) x = (f < 3 ? s.pos : f < 6 ? s.vel : s.acc)[3 * b + f % 3];
    else if (f < 13) x = s.Q[4 * b + f - 9];
    else x = (f < 16 ? s.vrot : s.arot)[3 * b + (f - 13) % 3];
    len = fmt_e(x, prec, false, cell);
  }
  const int L = conf_line(lane == 0 ? nullptr : cell, len, 23, o);
  if (lane == 0) lens[b] = L;
}

// 1 for the entries saveConf writes: dn < 0 or bonded (Rockable.cpp:3005-3029)
__global__ void k_conf_active(Scene s, int64_t* flag) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= s.ne) return;
  flag[e] = (s.dn[e] < 0.0 || s.bond[e] >= 0) ? 1 : 0;
}

// "i j type isub jsub n dn pos vel fn ft mom damp\n", the normal rounded
// toward zero (Rockable.cpp:569-575); line k of the active entries.  A warp
// takes 32 entries and writes the lines of the active ones among them.
__global__ void k_conf_entries(Scene s, const int64_t* pos, int prec, char* slots, int64_t* lens) {
  const int64_t e0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~(int64_t)31;
  const int lane = threadIdx.x & 31;
  const bool active = e0 + lane < s.ne && (s.dn[e0 + lane] < 0.0 || s.bond[e0 + lane] >= 0);
  for (unsigned m = __ballot_sync(0xffffffffu, active); m; m &= m - 1u) {
    const int64_t e = e0 + __ffs(m) - 1;
    const int64_t k = pos[e];
    char cell[kConfCell];
    int len = 0;
    if (lane < 5) {
      const uint32_t ts = s.etsub[e];
      len = fmt_i(lane == 0   ? s.ei[e]
                  : lane == 1 ? s.ej[e]
                  : lane == 2 ? tsub_type(ts)
                  : lane == 3 ? tsub_isub(ts)
                              : tsub_jsub(ts),
                  cell);
    } else if (lane < 22) {
      const int f = lane - 5;  // n 0-2, dn 3, pos 4-6, vel 7-9, fn 10, ft 11-13, mom 14-16 (then damp)
      double x;
      if (f < 3) x = s.gn[3 * e + f];
      else if (f == 3) x = s.dn[e];
      else if (f < 10) x = (f < 7 ? s.gpos : s.gvel)[3 * e + (f - 4) % 3];
      else if (f == 10) x = s.fn[e];
      else x = (f < 14 ? s.ft : s.mom)[3 * e + (f - 11) % 3];
      len = fmt_e(x, prec, f < 3, cell);
    } else if (lane == 22) {
      len = fmt_e(s.damp[e], prec, false, cell);
    }
    const int L = conf_line(cell, len, 23, slots + k * (int64_t)kConfEntrySlot);
    if (lane == 0) lens[k] = L;
  }
}

// line k of `slots` to out + ofs[k]: one warp per line
__global__ void k_conf_pack(const char* slots, int slot, const int64_t* ofs, const int64_t* lens, int64_t n,
                            char* out) {
  const int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (k >= n) return;
  const char* src = slots + k * (int64_t)slot;
  char* dst = out + ofs[k];
  const int64_t L = lens[k];
  for (int64_t q = lane; q < L; q += 32) dst[q] = src[q];
}

}  // namespace rk
