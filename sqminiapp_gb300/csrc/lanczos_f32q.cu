// lanczos_f32q.cu -- instantiations of the split-pass FP32 Lanczos kernel (kLayoutQuad) and its
// host-side sizes.
#include <algorithm>

#include "lanczos_quad.cuh"

namespace sq {

int lanczos_quad_threads(const LanczosParams &p) {
  // pitch/4 threads per row (pass A) or plane (pass B), zchunks ranges each (a pair: rows
  // over the owned planes, zchunks z-ranges; owned planes, ychunks y-ranges)
  // at least two warps: warp 0 builds the per-node image list while the others clear P and U
  const int groups = (p.layout & kLayoutPair)
                         ? std::max(p.ny * p.zchunks, lq::pair_u_planes(p.nz, p.zsplit) * p.ychunks)
                         : std::max(p.ny, p.nz) * p.zchunks;
  return std::max(64, 32 * (((p.pitch / 4) * groups + 31) / 32));
}

int lanczos_quad_block(const LanczosParams &p) {
  // every warp of the register budget (12 warps at up to 384 threads, 16 above): the passes
  // use lanczos_quad_threads of them, the list streams and the update all
  int t = lanczos_quad_threads(p);
  // at least as many as give the list items that its words hold (a cube of 3 x 69 x 69 points and one
  // range has a thread per column, of 69 planes)
  const int columns = p.pitch / 4 * p.ny;
  auto longest = [&](int threads) {
    const int chunks = lq::list_chunks(columns, p.nz, threads);
    return (p.nz + chunks - 1) / chunks;
  };
  while (t < kQuadMaxThreads && longest(t) > kQuadListPlanes) t += 32;
  if (t <= 256) return t;
  return t <= 384 ? 384 : kQuadMaxThreads;
}

size_t lanczos_quad_smem_bytes(const LanczosParams &p) {
  const bool pair = (p.layout & kLayoutPair) != 0;
  const size_t ps = lq::quad_plane_floats(p.ny, p.pitch);
  const int nlm = mask_nlm(kernel_mask(p.union_mask));
  const size_t pu[2] = {  // planes of P and of U
      (size_t)(pair ? lq::pair_p_planes(p.nz, p.zsplit) : lq::list_planes(p.nz)),
      (size_t)(pair ? lq::pair_u_planes(p.nz, p.zsplit) : lq::list_planes(p.nz))};
  size_t b = sizeof(float) * ps * (pu[0] + pu[1]);
  b += sizeof(float2) * (2 * lk::kMaxWarps + 128);           // partials and step sums
  b += sizeof(float4) * (size_t)p.max_img * ((nlm + 3) / 4);  // alpha
  if (pair)  // both CTAs' c, an 8-byte alignment, projector a_k partials, capacity flags
    b += sizeof(float) * 2 * (size_t)p.max_img * nlm + 8 + sizeof(float) * 2 * lk::kMaxWarps +
         sizeof(int) * 4;
  b += sizeof(int) * (4 * (size_t)p.max_img + 2 + 5 + lk::kMaxWarps);  // per-node lists
  b += 16 + sizeof(lq::ImgRow) * (size_t)p.max_img + sizeof(float4);   // image rows, a quad of zeros
  b += sizeof(float4) * (size_t)p.part_cap;
  const size_t scratch = lq::list_scratch_bytes(p.max_img, kQuadMaxThreads / 32);
  if (scratch > sizeof(float) * ps * pu[1]) b += scratch;  // list build, where U is too small for it
  return b;
}

static_assert(kQuadListRun == lq::kRun, "host and device agree on the list's units");
int lanczos_quad_list_chunks(int columns, int planes, int threads) {
  return lq::list_chunks(columns, planes, threads);
}

namespace {
int channels(const LanczosParams &p) {
  int n = 0;
  for (int l = 0; l < 4; l++) n += (kernel_mask(p.union_mask) >> l) & 1;
  return n;
}
size_t partial_float4(const LanczosParams &p) { return (mask_nlm(kernel_mask(p.union_mask)) + 3) / 4; }
}  // namespace

size_t lanczos_quad_unit_bytes(const LanczosParams &p) {
  return sizeof(float4) * (lq::kRun * channels(p) + 1);
}

size_t lanczos_quad_list_bytes(const LanczosParams &p) {
  return (size_t)p.list_batches * 32 * lanczos_quad_unit_bytes(p) +
         sizeof(float4) * partial_float4(p) * (size_t)p.part_total +
         sizeof(int2) * (size_t)p.max_img * kQuadMaxThreads;  // runs of every item
}

int lanczos_quad_place_partials(LanczosParams &p, int block, int smem_optin) {
  // part_total counts whole boxes; the units of the spheres in them are about half (2161 of 4608 on
  // a 27^3 cube).  A node with more keeps its partial sums in the scratch slice.
  p.part_cap = 0;
  const size_t base = lanczos_quad_smem_bytes(p), reserved = 1024, sm = (size_t)smem_optin + reserved;
  const size_t want = sizeof(float4) * partial_float4(p) * (size_t)(0.6 * p.part_total + 1);
  // CTAs on an SM by shared memory (the partial sums included) and by registers: 12 warps of the
  // 168-register kernels, one CTA of the others
  int ctas = 1;
  if (!(p.layout & kLayoutPair) && block <= 384)
    ctas = std::max(1, std::min(std::min(4, 12 / (block / 32)), (int)(sm / (base + want + reserved))));
  p.list_columns = ctas > 2 ? lq::kListColumns / 4 : lq::kListColumns / ctas;
  const size_t room = sm / ctas - reserved - base;
  p.part_cap = (int)(std::min(room, want) / sizeof(float4));
  return ctas;
}

// ---- quad tables ----
long long quad_table_float4(const TypeDesc &td) {
  return 4LL * __builtin_popcount(td.chan_mask) * lq::quad_table_channel(td);
}

namespace {
// One block row per table: for every shift, quads of the table's rows behind `shift` zeros, zeros where
// the point lies outside the support sphere; the planes and channels of a quad next to one another.
__global__ void quad_tables_kernel(const __grid_constant__ LanczosParams p, const QuadTable *__restrict__ tabs,
                                   const float *__restrict__ src, float4 *__restrict__ dst) {
  const QuadTable t = tabs[blockIdx.x];
  const TypeDesc &td = p.types[t.type];
  const int row = lq::quad_table_row(td), chan = lq::quad_table_channel(td);
  const int nch = __popc(td.chan_mask), fvol = td.fx * td.fy * td.fz;
  for (int e = threadIdx.x + blockDim.x * blockIdx.y; e < 4 * nch * chan; e += blockDim.x * gridDim.y) {
    const int shift = e / (nch * chan), r = e - shift * nch * chan, c = r % nch, lz = r / nch % td.fz;
    const int i = r / (nch * td.fz), q = i % row, ly = i / row;
    const float dy = fmaf(p.hyf, float(ly), t.oy), dz = fmaf(p.hzf, float(lz), t.oz);
    float v[4];
    for (int j = 0; j < 4; j++) {
      const int lx = 4 * q + j - shift;
      const float dx = fmaf(p.hxf, float(lx), t.ox);
      const bool in = lx >= 0 && lx < td.fx && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= td.support_r2_f32;
      v[j] = in ? src[t.src + (long long)c * fvol + (lz * td.fy + ly) * td.fx + lx] : 0.f;
    }
    dst[t.dst + e] = make_float4(v[0], v[1], v[2], v[3]);
  }
}
}  // namespace

cudaError_t launch_quad_tables(const LanczosParams &p, const QuadTable *tabs, int n, const float *src,
                               void *dst, cudaStream_t s) {
  quad_tables_kernel<<<dim3(n, 16), 256, 0, s>>>(p, tabs, src, (float4 *)dst);
  return cudaGetLastError();
}

size_t veff_quad_floats(const LanczosParams &p) { return 4 * (size_t)p.vq_copy_stride; }

namespace {
template <int MAXT, bool ISO>
cudaError_t launch_quad_mask(int mask, const LanczosParams &p, int grid, int block, size_t smem,
                             cudaStream_t s, const void *veffq, const ImageMeta *images,
                             const void *tables, void *proj_scratch, double *ab, int *status) {
  switch (mask) {
    case 3: return lq::launch_quad_variant<3, MAXT, ISO>(p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status);
    case 5: return lq::launch_quad_variant<5, MAXT, ISO>(p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status);
    case 6: return lq::launch_quad_variant<6, MAXT, ISO>(p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status);
    case 7: return lq::launch_quad_variant<7, MAXT, ISO>(p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status);
    default: return lq::launch_quad_variant<15, MAXT, ISO>(p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status);
  }
}
}  // namespace

// Two register budgets: up to 12 warps (3 per SM sub-partition: 168 registers a thread) and up
// to 16 warps (128).  Isotropic meshes (hx = hy = hz) share one set of stencil weights.
cudaError_t launch_lanczos_f32_quad(int mask, const LanczosParams &p, int grid, int block,
                                    size_t smem, cudaStream_t s, const void *veffq,
                                    const ImageMeta *images, const void *tables,
                                    void *proj_scratch, double *ab, int *status) {
  bool iso = true;
  for (int d = 0; d <= kStencilHalf; d++)
    iso = iso && p.cxf[d] == p.czf[d] && p.cyf[d] == p.czf[d];
  if (block <= 384)
    return iso ? launch_quad_mask<384, true>(mask, p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status)
               : launch_quad_mask<384, false>(mask, p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status);
  return iso ? launch_quad_mask<kQuadMaxThreads, true>(mask, p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status)
             : launch_quad_mask<kQuadMaxThreads, false>(mask, p, grid, block, smem, s, veffq, images, tables, proj_scratch, ab, status);
}

}  // namespace sq
