// Set-up, launch and selection of the pass-kernel variants of one grid size.
#include <string>

#include "../../include/mhdgb.h"
#include "ops.cuh"

namespace mhdgb {

OpsBase::~OpsBase() {
  if (tw_dev) cudaFree(tw_dev);
  for (auto& x : xv)
    if (x.table) cudaFree(x.table);
}

namespace {

int set_smem(const void* fn, size_t bytes) {
  if (bytes <= 48 * 1024) return MHD_OK;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return report_error(MHD_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
  return MHD_OK;
}

// Resident CTAs of a kernel on the whole device (persistent grid size); 0 when it does not fit.
int resident_ctas(const void* fn, int threads, size_t smem, int sms, int* out) {
  int per = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem);
  if (e != cudaSuccess) return report_error(MHD_ERR_CUDA, std::string("occupancy query: ") + cudaGetErrorString(e));
  *out = per * sms;
  return MHD_OK;
}

bool is_col(int cls) { return cls == KC_ZINV || cls == KC_YINV || cls == KC_YFWD || cls == KC_ZFWD; }
// in plane order the z classes carry the plane passes
bool plane_cls(int cls) { return cls == KC_ZINV || cls == KC_ZFWD; }
bool is_inv(int cls) { return cls == KC_ZINV || cls == KC_YINV; }

}  // namespace

// A variant's kernels are set up (attributes, occupancy, tables) when it is first asked for: a handle
// that runs on its defaults pays for those alone.
bool OpsBase::ready(XVariant& x) const {
  if (x.state) return x.state > 0;
  x.state = -1;
  const void* fn = x.tile_fn ? (const void*)x.tile_fn : (const void*)x.fn;
  x.smem = x.tile_fn ? x.tile_smem : sizeof(float2) * (size_t)x.groups * x.group_words(kxp);
  if ((int)x.smem > smem_limit) return false;
  if (x.build_table) {
    if (!x.table && cudaMalloc(&x.table, x.table_words * sizeof(uint32_t)) != cudaSuccess) {
      cudaGetLastError();
      x.table = nullptr;
      x.state = 0;  // asked for again, there may be memory
      table_rc = MHD_ERR_OOM;
      return false;
    }
    if (x.build_table(x.table)) {
      cudaGetLastError();
      table_rc = MHD_ERR_CUDA;
      return false;
    }
  }
  // max_carveout: the whole unified L1 / shared array as shared memory (two CTAs per SM fit only then)
  if (set_smem(fn, x.smem) ||
      (x.max_carveout && cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100) != cudaSuccess) ||
      resident_ctas(fn, x.threads, x.smem, sm_count, &x.ctas) || x.ctas == 0)
    return false;
  x.state = 1;
  return true;
}
bool OpsBase::ready(PlaneVariant& v, bool inv) const {
  int& state = inv ? v.state_inv : v.state_fwd;
  if (state) return state > 0;
  state = -1;
  if ((int)v.smem > smem_limit) return false;
  int ctas = 0;
  const void* main = inv ? (const void*)v.inv : (const void*)v.fwd;
  if (set_smem(main, v.smem) || resident_ctas(main, v.threads, v.smem, sm_count, &ctas) || ctas == 0) return false;
  if (inv)
    for (const void* f : {(const void*)v.stage, (const void*)v.stage_gen, (const void*)v.stage_hd})
      if (f && set_smem(f, v.smem)) return false;
  state = 1;
  return true;
}
bool OpsBase::ready(ColVariant& c, bool inv) const {
  int& state = inv ? c.state_inv : c.state_fwd;
  if (state) return state > 0;
  state = -1;
  if ((int)c.smem > smem_limit) return false;
  const void* f = inv ? (c.inv_pair ? (const void*)c.inv_pair : c.inv_tma ? (const void*)c.inv_tma : (const void*)c.inv)
                      : (c.fwd_pair ? (const void*)c.fwd_pair : c.fwd_tma ? (const void*)c.fwd_tma : (const void*)c.fwd);
  int& ctas = inv ? c.ctas_inv : c.ctas_fwd;
  if (set_smem(f, c.smem) || resident_ctas(f, c.threads, c.smem, sm_count, &ctas) || ctas == 0) return false;
  state = 1;
  return true;
}

int OpsBase::setup(const Geom& g) {
  if (g.kx != kept_kx_of(n) || g.kp != kept_kx_of(n) || g.kn != kept_kn_of(n))
    return report_error(MHD_ERR_INVALID, "kept-mode counts differ from the compiled pass plans");
  int rc = MHD_OK, dev = 0, sms = 0, smem_max = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return report_error(MHD_ERR_CUDA, std::string("device query: ") + cudaGetErrorString(e));
  e = cudaMalloc(&tw_dev, tw_host.size() * sizeof(float2));
  if (e != cudaSuccess) return report_error(MHD_ERR_OOM, std::string("twiddle tables: ") + cudaGetErrorString(e));
  e = cudaMemcpy(tw_dev, tw_host.data(), tw_host.size() * sizeof(float2), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return report_error(MHD_ERR_CUDA, std::string("twiddle upload: ") + cudaGetErrorString(e));
  sm_count = sms;
  smem_limit = smem_max;
  kxp = g.kxp;
  if (!cv.empty() && (cv[0].inv_tma || cv[0].inv_pair)) return report_error(MHD_ERR_INVALID, "the default column variant must not be TMA-fed");
  if ((rc = set_smem(planar ? (const void*)c2r_plane : (const void*)c2r, row_smem))) return rc;
  if ((rc = set_smem(planar ? (const void*)r2c_plane : (const void*)r2c, row_smem))) return rc;
  // the single-field transforms and a missing tensor map fall back to the first column variant
  if (!planar && (cv.empty() || !ready(cv[0], true) || !ready(cv[0], false)))
    return report_error(MHD_ERR_CUDA, "no pass-kernel variant fits on this device");
  // the default of each class is its first variant that fits on this device and names the class as its
  // own, else the first that fits
  for (int cls = 0; cls < kTunedClasses; ++cls) {
    int i = 0;
    while (i < variant_count(cls) && !(preferred(cls, i) && variant_ok(cls, i))) ++i;
    if (i == variant_count(cls))
      for (i = 0; i < variant_count(cls) && !variant_ok(cls, i);) ++i;
    if (i == variant_count(cls) && cls == KC_XFUSED && table_rc)
      return report_error(table_rc, table_rc == MHD_ERR_OOM ? "tensor-core tables: out of memory"
                                                            : "building the tensor-core DFT tables failed");
    if (i == variant_count(cls))
      return report_error(cls == KC_XFUSED && prec ? MHD_ERR_INVALID : MHD_ERR_CUDA,
                          cls == KC_XFUSED && prec ? "no x-row kernel of this precision form for this grid size"
                                                   : "no pass-kernel variant fits on this device");
    sel[cls] = i;
  }
  return MHD_OK;
}

// whether a variant names the class (and, in plane order, the capacity) as its own
bool OpsBase::preferred(int cls, int i) const {
  if (cls == KC_XFUSED) return true;  // one default for all capacities: a slot's results equal a single problem's bit for bit
  if (planar) return !plane_cls(cls) || (pv[i].pref >> (is_inv(cls) ? 0 : 1) >> (batch ? 2 : 0) & 1);
  return cv[i].pref & (cls == KC_ZINV ? kDefaultZinv : cls == KC_YINV ? kDefaultYinv : cls == KC_YFWD ? kDefaultYfwd : kDefaultZfwd);
}

int OpsBase::set_vp(int mode) {
  if (mode == vp) return MHD_OK;
  const int old = vp;
  vp = mode;
  for (int i = 0; i < (int)xv.size(); ++i)
    if (variant_ok(KC_XFUSED, i)) { sel[KC_XFUSED] = i; return MHD_OK; }
  vp = old;
  return report_error(MHD_ERR_INVALID, "no x-row kernel of this volume-penalisation form for this grid size");
}

int OpsBase::variant_count(int cls) const {
  if (cls == KC_XFUSED) return (int)xv.size();
  if (!is_col(cls)) return 0;
  if (planar) return plane_cls(cls) ? (int)pv.size() : 1;
  return (int)cv.size();
}

bool OpsBase::variant_ok(int cls, int i) const {
  if (i < 0 || i >= variant_count(cls)) return false;
  if (cls == KC_XFUSED)  // this problem's precision, penalty form, field set and layout only
    return xv[i].prec == prec && xv[i].vp == vp && xv[i].hd == hd && xv[i].plane == planar && ready(xv[i]);
  if (planar) return !plane_cls(cls) || ready(pv[i], is_inv(cls));
  return ready(cv[i], is_inv(cls));
}

std::string OpsBase::variant_name(int cls, int i) const {
  if (i < 0 || i >= variant_count(cls)) return "";
  if (cls == KC_XFUSED) return xv[i].name;
  if (planar) return plane_cls(cls) ? pv[i].name : std::string("plane");
  return cv[i].name;
}

int OpsBase::select(int cls, int i) {
  if (cls < 0 || cls >= kTunedClasses || !variant_ok(cls, i))
    return report_error(MHD_ERR_INVALID, "no such kernel variant (class " + std::to_string(cls) + ", index " +
                                             std::to_string(i) + ")");
  sel[cls] = i;
  return MHD_OK;
}

int OpsBase::select_by_name(int cls, const std::string& name) {
  for (int i = 0; i < variant_count(cls); ++i)
    if (variant_name(cls, i) == name) return select(cls, i);
  return report_error(MHD_ERR_INVALID, "no kernel variant named " + name);
}

void OpsBase::col(int cls, const ColArgs& a, const Geom& g, int outer, int nf, BatchRef br,
                  cudaStream_t s, const TmaPass* tp, const TmaPass* to) const {
  const ColVariant& sv = cv[sel[cls]];
  const bool in = tp && tp->ok, out = to && to->ok;
  const ColVariant& c = (sv.inv_tma && !in) || (sv.inv_pair && !(in && out)) ? cv[0] : sv;
  const bool inv = is_inv(cls);
  const ColWork w{(g.kx + c.tx - 1) / c.tx, outer, nf, inv ? g.k2 : n};
  const long long total = (long long)br.most * w.tiles_x * w.outer * w.nf;
  const int ctas = inv ? c.ctas_inv : c.ctas_fwd;
  const int grid = (int)(total < ctas ? total : ctas);
  if (c.inv_pair) {
    (inv ? c.inv_pair : c.fwd_pair)<<<grid, c.threads, c.smem, s>>>(a, g, w, br, tw_dev + c.tw, tp->map, tp->tc, to->map, to->tc, tp->err);
    return;
  }
  if (c.inv_tma) {
    (inv ? c.inv_tma : c.fwd_tma)<<<grid, c.threads, c.smem, s>>>(a, g, w, br, tw_dev + c.tw, tp->map, tp->tc, tp->err);
    return;
  }
  const ColFn f = inv ? c.inv : c.fwd;
  f<<<grid, c.threads, c.smem, s>>>(a, g, w, br, tw_dev + c.tw);
}

void OpsBase::plane_forward(const PlaneArgs& a, const Geom& g, int nslots, BatchRef br, cudaStream_t s) const {
  const PlaneVariant& v = pv[sel[KC_ZFWD]];
  v.fwd<<<dim3(g.kx, nslots, br.most), v.threads, v.smem, s>>>(a, g, br, tw_dev + v.tw);
}

void OpsBase::plane_inverse(const PlaneArgs& a, const Geom& g, int nf, BatchRef br, cudaStream_t s) const {
  const PlaneVariant& v = pv[sel[KC_ZINV]];
  v.inv<<<dim3(g.kx, nf, br.most), v.threads, v.smem, s>>>(a, br, tw_dev + v.tw);
}

void OpsBase::plane_stage(const RkArgs& a, const PlaneArgs& pa, const Geom& g, int nf, bool inv, BatchRef br,
                          cudaStream_t s) const {
  const PlaneVariant& v = pv[sel[KC_ZINV]];
  const PlaneStageFn f = hd ? v.stage_hd : (a.vpen || a.forced) ? v.stage_gen : v.stage;
  f<<<dim3(g.kx, nf, br.most), v.threads, v.smem, s>>>(a, pa, g, br, inv ? 1 : 0, tw_dev + v.tw);
}

void OpsBase::x_fused(float2* pool, const Geom& g, long long rowstride, long long slot, long long istride,
                      BatchRef br, unsigned int* vmax, VpRef vp, int* err, cudaStream_t s, const TmaPass* tp) const {
  const XVariant* sv = &xv[sel[KC_XFUSED]];
  if (sv->tile_fn && !(tp && tp->ok))  // no tensor map: the first variant of this form without one
    for (size_t i = 0; i < xv.size(); ++i)
      if (variant_ok(KC_XFUSED, (int)i) && !xv[i].tile_fn) { sv = &xv[i]; break; }
  const XVariant& x = *sv;
  if (x.tile_fn) {
    const long long tiles = (long long)br.most * n * n / x.rpg;
    x.tile_fn<<<(unsigned)(tiles < x.ctas ? tiles : x.ctas), x.threads, x.smem, s>>>(tp->map, tp->err, br, tw_dev + x.tw,
                                                                                    tw_dev + x.twr, vmax, vp);
    return;
  }
  const long long groups = (long long)br.most * n * n / x.rpg;
  const long long need = (groups + x.groups - 1) / x.groups;
  const int grid = (int)(need < x.ctas ? need : x.ctas);
  const float2* t1 = x.table ? reinterpret_cast<const float2*>(x.table) : tw_dev + x.tw;
  const float2* t2 = x.table ? nullptr : tw_dev + x.twr;
  x.fn<<<grid, x.threads, x.smem, s>>>(pool, g, rowstride, slot, istride, br, t1, t2, vmax, vp, err);
}

int OpsBase::x_device_error() const {
  const XVariant& x = xv[sel[KC_XFUSED]];
  if (!x.table || x.err_word < 0) return 0;
  uint32_t e = 0;
  if (cudaMemcpy(&e, x.table + x.err_word, sizeof(e), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  return e != 0;
}

void OpsBase::x_c2r(const float2* src, float* dst, const Geom& g, long long srow, float scale, cudaStream_t s) const {
  const long long pairs = (long long)n * n / 2;
  (planar ? c2r_plane : c2r)<<<(unsigned)(pairs / rows), row_threads, row_smem, s>>>(src, dst, g, srow, scale, tw_dev + row_tw);
}

void OpsBase::x_r2c(const float* src, float2* dst, const Geom& g, long long drow, cudaStream_t s) const {
  const long long pairs = (long long)n * n / 2;
  (planar ? r2c_plane : r2c)<<<(unsigned)(pairs / rows), row_threads, row_smem, s>>>(src, dst, g, drow, tw_dev + row_tw);
}

}  // namespace mhdgb
