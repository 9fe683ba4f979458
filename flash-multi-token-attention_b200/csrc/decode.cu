// Instantiations and launcher of the decode kernel and the split combine.
#include "decode.cuh"
#include "launch_util.cuh"

namespace fmta {

namespace {

template <int D, int NR, int CKP, bool PAGED, bool A32>
cudaError_t launch_decode_t(const DecodeParams& p, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.k_splits * p.n_sub, p.H, p.B); cfg.blockDim = dim3(kDecWarps * 32); cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  if (pdl_enabled()) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  const unsigned cl = p.fused ? p.k_splits * p.n_sub : p.n_sub;
  if (cl > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cl;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  return cudaLaunchKernelEx(&cfg, decode_kernel<D, NR, CKP, PAGED, A32>, p);
}

template <int D, int NR, int CKP>
cudaError_t launch_decode_p(const DecodeParams& p, cudaStream_t stream) {
  constexpr bool kWide = D >= 64;            // head dim 32 has no 32-byte loads
  const bool a32 = ((reinterpret_cast<uintptr_t>(p.K) | reinterpret_cast<uintptr_t>(p.V)) & 31) == 0;
  if (kWide && !a32) return p.block_table ? launch_decode_t<D, NR, CKP, true, !kWide>(p, stream) : launch_decode_t<D, NR, CKP, false, !kWide>(p, stream);
  return p.block_table ? launch_decode_t<D, NR, CKP, true, true>(p, stream) : launch_decode_t<D, NR, CKP, false, true>(p, stream);
}
template <int D, int NR>
cudaError_t launch_decode_c(const DecodeParams& p, cudaStream_t stream) {
  if (p.ck <= 9) return launch_decode_p<D, NR, 9>(p, stream);
  if (p.ck == 11) return launch_decode_p<D, NR, 11>(p, stream);
  return launch_decode_p<D, NR, 17>(p, stream);
}
template <int D>
cudaError_t launch_decode_d(const DecodeParams& p, cudaStream_t stream) {
  return (p.q_len < p.cq ? p.q_len : p.cq) > 8 ? launch_decode_c<D, 4>(p, stream) : launch_decode_c<D, 2>(p, stream);
}

}  // namespace

cudaError_t launch_decode(const DecodeParams& p_, cudaStream_t stream) {
  DecodeParams p = p_;
  // A split is the caller's unit, so few (batch, head) pairs and few splits would leave SMs without work: a split is then
  // divided over up to 8 CTAs (one cluster), as long as each keeps 256 keys (8 steps of its 4 warps' 32-key blocks; below
  // that the merge costs what the division gives).
  const long ctas = (long)p.B * p.H * p.k_splits;
  const int kps = decode_keys_per_split(p.Nk, p.k_splits);
  p.n_sub = 1;
  while (p.n_sub < 8 && ctas * p.n_sub < 2 * kSMs && kps / (2 * p.n_sub) >= 256) p.n_sub *= 2;
  // One split needs no merge of splits; up to eight CTAs per (batch, head) on a GPU that is not full merge in their
  // cluster, which saves the second launch (a full GPU keeps the free placement of single CTAs).
  p.fused = p.k_splits == 1 || (p.k_splits * p.n_sub <= 8 && ctas * p.n_sub <= 2 * kSMs);
  cudaError_t e;
  {
    ScopedKernelTimer timer_(kKernDecode, stream);
    if (p.d == 32) e = launch_decode_d<32>(p, stream);
    else if (p.d == 64) e = launch_decode_d<64>(p, stream);
    else if (p.d == 128) e = launch_decode_d<128>(p, stream);
    else return cudaErrorInvalidValue;
  }
  if (e != cudaSuccess || p.fused) return e;
  return launch_pdl(combine_splits_kernel, dim3(p.B * p.H), dim3(128), 0, stream, p.O_splits, p.M_splits, p.L_splits, p.k_splits, p.d);
}

cudaError_t launch_kv_append_paged(void* Kpool, void* Vpool, const int* block_table, const int* seq_lens,
                                   const void* Knew, const void* Vnew, int B, int H, int n_new, int d, int page_size,
                                   int page_shift, int max_pages, cudaStream_t stream) {
  const int chunks = H * n_new * (d / 8);
  dim3 grid((chunks + 127) / 128, 1, B), block(128);
  bf16* kp = reinterpret_cast<bf16*>(Kpool); bf16* vp = reinterpret_cast<bf16*>(Vpool);
  const bf16* kn = reinterpret_cast<const bf16*>(Knew); const bf16* vn = reinterpret_cast<const bf16*>(Vnew);
  if (d == 32) return launch_pdl(kv_append_paged_kernel<32>, grid, block, 0, stream, kp, vp, block_table, seq_lens, kn, vn, H, n_new, page_size, page_shift, max_pages);
  else if (d == 64) return launch_pdl(kv_append_paged_kernel<64>, grid, block, 0, stream, kp, vp, block_table, seq_lens, kn, vn, H, n_new, page_size, page_shift, max_pages);
  else if (d == 128) return launch_pdl(kv_append_paged_kernel<128>, grid, block, 0, stream, kp, vp, block_table, seq_lens, kn, vn, H, n_new, page_size, page_shift, max_pages);
  return cudaErrorInvalidValue;
}

}  // namespace fmta
