// Internal host interfaces shared between the library's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "common.cuh"
#include "sort.cuh"

namespace crt {

// Once per device: the stream-ordered pool keeps what is freed.
void init_device();

int tree_levels(int64_t n, int fanout, std::vector<int64_t>& lv);

int build_tree(const float* in_xmin, const float* in_ymin, const float* in_xmax,
               const float* in_ymax, const int* in_id, int64_t n, int fanout, float* out_xmin,
               float* out_ymin, float* out_xmax, float* out_ymax, int* out_id, float* nxmin,
               float* nymin, float* nxmax, float* nymax, int* npos, int* nlen,
               cudaStream_t stream);

int pairs_canonicalize(int32_t* fid, int32_t* tid, int64_t n, cudaStream_t stream);
int pairs_digest(const int32_t* fid, const int32_t* tid, int64_t n, int64_t window_base,
                 int64_t nq, int64_t* d_counts, uint64_t* d_hashes, int64_t* d_bad,
                 cudaStream_t stream);

// Query entry used by the C ABI.
int query_into(const crt_rtree_f32& rt, const crt_bbox_f32& rbox, const crt_bbox_f32& qbox,
               int32_t* fid, int32_t* tid, int64_t capacity, crt_query_result* d_result,
               int64_t* d_offsets, const crt_query_opts& opts, cudaStream_t stream);
int64_t query_capacity(int64_t pairs, const crt_query_opts& opts);
bool query_dense_fits(int64_t nbox, int fanout);
int query_dense(const crt_rtree_f32& rt, const crt_bbox_f32& rbox, const crt_bbox_f32& qbox,
                int32_t* fid, int32_t* tid, int64_t cap, int64_t* pairs, cudaStream_t stream);

// Host parser of the reference's MBR text format (io.cu), with the rules of
// readMBR's fscanf(fp, "%f,%f,%f,%f,%d,%d,%d\n", ...): one record at p (the
// position after it and the whitespace that follows, or nullptr where fscanf
// reads fewer than seven fields), the box readMBR makes of its four numbers,
// and whole texts: scan_mbr_text reads up to `limit` records (limit < 0:
// all) in fscanf's order, stopping at the end of the text or at a malformed
// record; read_mbr_text does so into caller arrays (statuses and *n_read as
// crt_read_mbr_csv).
const char* parse_mbr_record(const char* p, const char* end, float v[4], int& id);
void mbr_box(const float v[4], float r, float* xmin, float* ymin, float* xmax, float* ymax);
struct MbrRecords {
  std::vector<float> v[4];  // xmin, ymin, xmax, ymax
  std::vector<int32_t> id;
  int64_t count = 0;
  bool malformed = false;  // stopped at a record fscanf cannot read
};
void scan_mbr_text(const char* base, size_t len, int64_t limit, float r, MbrRecords& out);
int read_mbr_text(const char* base, size_t len, int64_t n, float r, float* xmin, float* ymin,
                  float* xmax, float* ymax, int32_t* id, int64_t* n_read);

}  // namespace crt
