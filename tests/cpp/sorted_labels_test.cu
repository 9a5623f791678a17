// sorted_labels_test.cu -- sorted_kinds() (gbx_sort.cu) over a hand-made
// table: with every key in it the first row of each group comes back; with a
// key missing the status says so (the groupby call turns that into an error).
// Linked with the library's objects; prints one line per case and "0 failure(s)".
#include <cuda_runtime.h>

#include <cstdio>
#include <vector>

#include "../../cudf_b200/csrc/gbx_host.hpp"
#include "../../cudf_b200/csrc/gbx_kernels.hpp"
#include "../../cudf_b200/csrc/gbx_sort.hpp"
#include "../../include/gbx.h"

using namespace gbx;

namespace {

template <class T>
T* upload(const std::vector<T>& h)
{
  void* d = nullptr;
  if (cudaMalloc(&d, h.size() * sizeof(T)) != cudaSuccess ||
      cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess)
    return nullptr;
  return static_cast<T*>(d);
}

// n rows of keys {7, 11, all ones} (row % 3), of which the table holds the first `known`.
int run(int64_t n, int known)
{
  const long long words[3] = {7, 11, -1};
  const uint64_t cap       = 64;
  const uint32_t slots[3]  = {5, 9, static_cast<uint32_t>(cap)};
  std::vector<long long> keys(n), vals(n);
  for (int64_t r = 0; r < n; ++r) keys[r] = words[r % 3], vals[r] = 100 + r;
  std::vector<uint64_t> tkeys(cap + 1, kEmptyWord);
  std::vector<uint32_t> map(slots, slots + known);
  for (int i = 0; i < known; ++i) tkeys[slots[i]] = static_cast<uint64_t>(words[i]);

  SortedKindsArgs a{};
  KeyCol& kc        = a.plan.key.cols[0];
  a.plan.key.ncols  = 1;
  a.plan.key.nwords = 1;
  kc.data           = upload(keys);
  kc.width          = 8;
  a.plan.nchan      = 1;
  Channel& ch       = a.plan.chan[0];
  ch.data           = upload(vals);
  ch.ptype          = P_I64;
  a.table.keys      = upload(tkeys);
  a.table.cap       = cap;
  a.map             = upload(map);
  a.num_groups      = known;
  a.n               = n;
  a.max_probes      = static_cast<uint32_t>(cap);
  a.status          = upload(std::vector<int32_t>{0, 0});
  a.table.status    = a.status;
  a.num_sms         = current_device().num_sms;
  SortedOut o{};
  o.kind        = GBX_AGG_NTH_ELEMENT;
  o.null_policy = GBX_NULL_INCLUDE;
  o.out_width   = 8;
  o.data        = upload(std::vector<long long>(3, 0));
  o.mask        = upload(std::vector<uint32_t>(1, 0));
  o.null_count  = upload(std::vector<unsigned long long>(1, 0));
  a.outs.push_back(o);
  Alloc alloc;
  int32_t status = -1;
  long long got[3] = {0, 0, 0};
  {
    Scratch sc(&alloc);
    a.scratch    = &sc;
    int launches = 0;
    sorted_kinds(a, &launches);
  }
  if (cudaMemcpy(&status, a.status, 4, cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(got, o.data, sizeof(got), cudaMemcpyDeviceToHost) != cudaSuccess)
    return 1;
  bool ok = (status & S_TABLE_FULL) == (known < 3 ? S_TABLE_FULL : 0);
  for (int i = 0; i < known; ++i) ok = ok && got[i] == 100 + i;
  std::printf("%s: %lld rows, %d of 3 keys in the table, status %d\n", ok ? "ok" : "FAILED",
              static_cast<long long>(n), known, status);
  return ok ? 0 : 1;
}

}  // namespace

int main()
{
  int failures = 0;
  // the label table read through L1, and in shared memory (from 2^20 rows on)
  for (int64_t n : {int64_t(5000), (int64_t(1) << 20) + 3})
    for (int known = 1; known <= 3; ++known) failures += run(n, known);
  std::printf("%d failure(s)\n", failures);
  return failures ? 1 : 0;
}
