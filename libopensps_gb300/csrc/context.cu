// Context setup: the libraries of the data root, their device tables, the contraction's basis operand, and the
// parameter table of the C API.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <iterator>
#include <sstream>
#include "context.h"
#include "datalib.h"

namespace sps {

// ---------------------------------------------------------------------------------------------- parameters
// The float parameters of the reference's parameter registry (src/core/opensps_batch_registry.f90:103-115) with
// their defaults (src/core/opensps_types.f90:32-45); id >= 0 for those this path takes per model.
static const ParamInfo PARAMS[] = {
    {"dust1", PF_DUST1, 0.0}, {"dust2", PF_DUST2, 0.0}, {"dust3", PF_DUST3, 0.0},
    {"dust_index", PF_DUST_INDEX, -0.7}, {"dust1_index", PF_DUST1_INDEX, -1.0},
    {"frac_nodust", PF_FRAC_NODUST, 0.0}, {"frac_obrun", PF_FRAC_OBRUN, 0.0}, {"zred", PF_ZRED, 0.0},
    {"igm_factor", PF_IGM_FACTOR, 1.0}, {"sigma_smooth", PF_SIGMA_SMOOTH, 0.0}, {"dust_tesc", PF_DUST_TESC, 7.0},
    {"logzsol", PF_LOGZSOL, 0.0}, {"tage", PF_TAGE, 0.0}, {"tau", PF_TAU, 1.0},
    {"min_wave_smooth", PF_MIN_WAVE_SMOOTH, 1.0e3}, {"max_wave_smooth", PF_MAX_WAVE_SMOOTH, 1.0e4},
    {"const", PF_CONST, 0.0}, {"fburst", PF_FBURST, 0.0}, {"tburst", PF_TBURST, 11.0},
    {"sf_start", PF_SF_START, 0.0}, {"sf_trunc", PF_SF_TRUNC, 0.0}, {"imf1", PF_IMF1, 1.3},
    {"imf2", PF_IMF2, 2.3}, {"imf3", PF_IMF3, 2.3}, {"duste_qpah", PF_DUSTE_QPAH, 3.5},
    {"duste_umin", PF_DUSTE_UMIN, 1.0}, {"duste_gamma", PF_DUSTE_GAMMA, 0.01}, {"fagn", PF_FAGN, 0.0},
    {"agn_tau", PF_AGN_TAU, 10.0}, {"sf_slope", PF_SF_SLOPE, 0.0},
    {"vdmc", PF_VDMC, 0.08}, {"mdave", PF_MDAVE, 0.5},
    // known to the reference, not varied per model by this path (gas_logz and gas_logu are: the nebular continuum;
    // mwr and uvb are, by the batch, with dust_type 1)
    {"afe", -1, 0.0}, {"fbhb", -1, 0.0}, {"sbss", -1, 0.0}, {"agb", -1, 1.0},
    {"pagb", -1, 1.0}, {"redgb", -1, 1.0}, {"delt", -1, 0.0}, {"dell", -1, 0.0}, {"imf_lower_limit", -1, 0.08},
    {"imf_upper_limit", -1, 120.0}, {"masscut", -1, 150.0}, {"agb_dust", -1, 1.0}, {"pmetals", -1, 0.02},
    {"fcstar", -1, 1.0}, {"frac_xrb", -1, 1.0}, {"dust_clumps", -1, -99.0}, {"uvb", PF_UVB, 1.0}, {"mwr", PF_MWR, 3.1},
    {"gas_logu", PF_GAS_LOGU, -2.0},
    {"gas_logz", PF_GAS_LOGZ, 0.0}, {"gas_logn", -1, 2.0}, {"gas_logno", -1, 0.0}, {"gas_logco", -1, 0.0},
    {"sfh", -1, 0.0}, {"zmet", -1, 1.0}, {"evtype", -1, -1.0},
    {"wgp1", -1, 1.0}, {"wgp2", -1, 1.0}, {"wgp3", -1, 1.0}, {"compute_mags", -1, 1.0},
    {"compute_indices", -1, 1.0},
};

const ParamInfo *find_param(const char *name) {
    if (!name) return nullptr;
    for (const auto &p : PARAMS)
        if (std::strcmp(p.name, name) == 0) return &p;
    return nullptr;
}

// ---------------------------------------------------------------------------------------------- errors
static std::mutex g_err_mu;
static int g_err_status = 0;
static std::string g_err_msg;

void set_error(int status, const std::string &msg) {
    std::lock_guard<std::mutex> lk(g_err_mu);
    g_err_status = status;
    g_err_msg = msg;
}
void get_error(int *status, std::string *msg) {
    std::lock_guard<std::mutex> lk(g_err_mu);
    *status = g_err_status;
    *msg = g_err_msg;
}
void clear_error() {
    std::lock_guard<std::mutex> lk(g_err_mu);
    g_err_status = 0;
    g_err_msg.clear();
}

// ---------------------------------------------------------------------------------------------- bf16
uint16_t f32_to_bf16_bits(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    if ((u & 0x7fffffffu) > 0x7f800000u) return (uint16_t)((u >> 16) | 0x40);   // NaN
    u += 0x7fffu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}
float bf16_bits_to_f32(uint16_t b) {
    uint32_t u = (uint32_t)b << 16;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

// ---------------------------------------------------------------------------------------------- TMA maps
typedef CUresult (*PFN_encodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                    const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode_fn() {
    static PFN_encodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeTiled>(p);
    });
    return fn;
}

// A 2-D bf16 tensor map over a row-major [outer][inner] array, box box_outer x box_inner with the 128-byte swizzle;
// elements outside the array read as zero.
cudaError_t encode_tmap_2d_bf16(CUtensorMap *m, const void *ptr, uint64_t inner, uint64_t outer, uint32_t box_inner,
                                uint32_t box_outer) {
    return encode_tmap_2d_16(m, ptr, inner, outer, box_inner, box_outer, false);
}
// The same over 16-bit elements that are bf16 (f16 = false) or f16.
cudaError_t encode_tmap_2d_16(CUtensorMap *m, const void *ptr, uint64_t inner, uint64_t outer, uint32_t box_inner,
                              uint32_t box_outer, bool f16) {
    return encode_tmap_2d_16s(m, ptr, inner, outer, inner, box_inner, box_outer, f16);
}
// The same with rows row_elems elements apart (a column range of a wider matrix).
cudaError_t encode_tmap_2d_16s(CUtensorMap *m, const void *ptr, uint64_t inner, uint64_t outer, uint64_t row_elems,
                               uint32_t box_inner, uint32_t box_outer, bool f16) {
    PFN_encodeTiled fn = get_encode_fn();
    if (!fn) return cudaErrorNotSupported;
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_elems * 2};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t es[2] = {1, 1};
    CUresult r = fn(m, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                    const_cast<void *>(ptr), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------------------------- data root
std::string data_root() {
    const char *e = std::getenv("OPENSPS_DATA_HOME");
    if (e && *e) return std::string(e);
    return std::string();
}

static bool read_f64(const std::string &path, std::vector<double> &out, size_t count) {
    std::ifstream f(path, std::ios::binary);
    if (!f) return false;
    out.resize(count);
    f.read(reinterpret_cast<char *>(out.data()), (std::streamsize)(count * sizeof(double)));
    return (size_t)f.gcount() == count * sizeof(double);
}

// A minimal reader of the manifest's integer fields ("key": value).
static bool manifest_int(const std::string &text, const char *key, long long &v) {
    std::string k = std::string("\"") + key + "\"";
    size_t p = text.find(k);
    if (p == std::string::npos) return false;
    p = text.find(':', p);
    if (p == std::string::npos) return false;
    v = std::strtoll(text.c_str() + p + 1, nullptr, 10);
    return true;
}
static bool manifest_double(const std::string &text, const char *key, double &v) {
    std::string k = std::string("\"") + key + "\"";
    size_t p = text.find(k);
    if (p == std::string::npos) return false;
    p = text.find(':', p);
    if (p == std::string::npos) return false;
    v = std::strtod(text.c_str() + p + 1, nullptr);
    return true;
}

Context::~Context() {
    for (auto &kv : basis_cache) {
        kv.second->release();
        delete kv.second;
    }
    d_ion.release(); d_pix.release(); d_wl.release(); d_igm_a.release(); d_do_band.release(); d_cb_hi.release(); d_cb_lo.release();
    d_lam.release(); d_lnlam.release(); d_mass.release(); d_llin.release(); d_zt.release(); d_dl.release();
    d_wz.release(); d_params.release(); d_sums.release(); d_zinfo.release(); d_dist.release(); d_fband.release();
    d_mags.release(); d_spec64.release(); d_whi.release(); d_wlo.release(); d_mpar.release(); d_spec.release();
    d_status.release(); d_young.release(); d_old.release(); d_eml.release(); d_eml_lum.release(); d_eml_kidx.release();
    d_bc.release(); d_bmeta.release(); d_bchunk.release(); d_mags_bar.release(); d_spec_bar.release(); d_mass_bar.release();
    d_lbol_bar.release(); d_cscale.release(); d_pbar.release(); d_wzbar.release(); d_ybh.release(); d_ybl.release();
    d_obh.release(); d_obl.release(); d_wzb32.release(); d_apar.release();
    d_logage.release(); d_lz.release(); d_lbol.release(); d_sfhpar.release(); d_wgiven.release(); d_w.release();
    d_sfh_scratch.release(); d_lblend.release(); d_sfr.release(); d_wbar.release(); d_dual.release(); d_sfhtab.release(); d_user_imf.release();
    ops.release(); dustem.release(); agn.release(); neb.release(); d_alpha.release(); d_vhi.release(); d_vlo.release(); d_yo.release(); d_vpart.release();
    d_spart.release(); d_vflag.release(); d_vbar.release(); d_apart.release(); d_ix_hi.release(); d_ix_lo.release(); d_ipart.release(); d_sfh_mtab.release(); d_ix_const.release(); d_ix_dln.release(); d_fold.release(); d_dem.release(); d_w64.release(); d_y64.release(); d_bc64.release(); d_igm_a64.release();
    fp64_release(*this);
    emu.release();
    if (pinned_spec) cudaFreeHost(pinned_spec);
    if (pinned_par) cudaFreeHost(pinned_par);
    pinned_par = nullptr;
    pinned_par_n = 0;
    if (pinned_dem) cudaFreeHost(pinned_dem);
    pinned_dem = nullptr;
    pinned_dem_n = 0;
    if (pinned_sums) cudaFreeHost(pinned_sums);
    pinned_sums = nullptr;
    pinned_sums_n = 0;
    if (pinned_fold) cudaFreeHost(pinned_fold);
    pinned_fold = nullptr;
    pinned_fold_n = 0;
    if (pinned_sfh) cudaFreeHost(pinned_sfh);
    pinned_sfh = nullptr;
    pinned_sfh_n = 0;
    if (pinned_sfhout) cudaFreeHost(pinned_sfhout);
    pinned_sfhout = nullptr;
    pinned_sfhout_n = 0;
    if (pinned_mags) cudaFreeHost(pinned_mags);
    pinned_mags = nullptr;
    pinned_mags_n = 0;
    for (int i = 0; i < NCHUNK_EV; ++i) {
        if (chunk_ev[i]) cudaEventDestroy(chunk_ev[i]);
        chunk_ev[i] = nullptr;
        if (mag_ev[i]) cudaEventDestroy(mag_ev[i]);
        mag_ev[i] = nullptr;
    }
    for (int s = 0; s < 2; ++s)
        for (int i = 0; i < NPROF; ++i) if (prof_ev[s][i]) cudaEventDestroy(prof_ev[s][i]);
    if (par_ev) cudaEventDestroy(par_ev);
    par_ev = nullptr;
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_params) cudaEventDestroy(ev_params);
    if (ev_sums) cudaEventDestroy(ev_sums);
    if (ev_contract) cudaEventDestroy(ev_contract);
    if (side) cudaStreamDestroy(side);
    if (side2) cudaStreamDestroy(side2);
    if (side3) cudaStreamDestroy(side3);
    if (side4) cudaStreamDestroy(side4);
    if (ev_cot) cudaEventDestroy(ev_cot);
    if (ev_w0) cudaEventDestroy(ev_w0);
    if (ev_w1) cudaEventDestroy(ev_w1);
    if (stream) cudaStreamDestroy(stream);
}

// Madau (1995) wavelength factors of the IGM optical depth (src/physics/opensps_cosmology.f90:466-494).
static void igm_pixel_terms(double w, double *a) {
    static const double LYW[17] = {1215.67, 1025.72, 972.537, 949.743, 937.803, 930.748, 926.226, 923.150, 920.963,
                                   919.352, 918.129, 917.181, 916.429, 915.824, 915.329, 914.919, 914.576};
    static const double LYC[17] = {0.0036, 0.0017, 0.0011846, 0.0009410, 0.0007960, 0.0006967, 0.0006236, 0.0005665,
                                   0.0005200, 0.0004817, 0.0004487, 0.0004200, 0.0003947, 0.000372, 0.000352,
                                   0.0003334, 0.00031644};
    for (int k = 0; k < 6; ++k) a[k] = 0.0;
    if (w < LYW[0]) {
        double ser = 0.0;
        for (int i = 0; i < 17; ++i)
            if (w < LYW[i]) ser += LYC[i] * std::pow(LYW[i], -3.46);
        a[0] = ser * std::pow(w, 3.46);
        a[1] = 0.0017 * std::pow(w / LYW[0], 1.68);
    }
    if (w < 911.75) {
        const double s = w / 911.75;
        a[2] = 0.25 * std::pow(s, 3.0) * (1.0 - std::pow(s, 0.46));
        a[3] = 9.4 * std::pow(s, 1.5) * (1.0 - std::pow(s, 0.18));
        a[4] = -0.7 * std::pow(s, 3.0) * (std::pow(s, -1.32) - 1.0);
        a[5] = -0.023 * (1.0 - std::pow(s, 1.68));
    }
}

// The cosmology table of update_cosmology_table (src/physics/opensps_cosmology.f90:244-300): 500 scale factors,
// luminosity distance [pc] by a 10000-point trapezoid.
static void cosmology_table(double h0, double om0, double ol0, std::vector<double> &zt, std::vector<double> &dl) {
    zt.resize(500);
    dl.resize(500);
    const double dh = ((C_LIGHT * 1.0e-13) / h0) * 1.0e6;
    for (int i = 1; i <= 500; ++i) {
        const double a = (double)(i - 1) / 499.0 * (1.0 - 1.0 / 1001.0) + 1.0 / 1001.0;
        const double z = 1.0 / a - 1.0;
        zt[i - 1] = z;
        double d = 0.0;
        if (z > 0.0) {
            const int N = 10000;
            const double dz = z / (double)(N - 1);
            double prev = 1.0 / std::sqrt(om0 + ol0), sum = 0.0;
            for (int k = 2; k <= N; ++k) {
                const double zc = (double)(k - 1) * dz;
                const double now = 1.0 / std::sqrt(om0 * std::pow(1.0 + zc, 3) + ol0);
                sum += 0.5 * dz * (prev + now);
                prev = now;
            }
            d = (1.0 + z) * dh * sum;
        }
        dl[i - 1] = d;
    }
}

template <class T>
static cudaError_t upload(DevBuf<T> &b, const T *src, size_t n) {
    cudaError_t e = b.reserve(n);
    if (e != cudaSuccess) return e;
    return cudaMemcpy(b.p, src, sizeof(T) * n, cudaMemcpyHostToDevice);
}

// The dust emission templates from the data root's dust_dl07 dataset (the reference reads its Draine & Li files at
// setup; here the synthetic stand-in): q_PAH and U_min grids, the templates on the context's wavelength grid, and
// the per-pixel frequency trapezoid weights of the energy sums (dust_emission_reductions' wt, the grid's
// prepare_batch_grid :262-265).
int dustem_load(Context &c, std::string &err) {
    if (c.dustem.ready) return 0;
    DustEmission &d = c.dustem;
    const std::string root = data_root();
    long long nq = 0, nu = 0, ns = c.nspec;
    std::vector<float> tab;
    if (datalib_available(root, "dust_emission", c.dust_emission_lib)) {
        // the standard format's dust_emission/<name> library, interpolated onto the grid
        std::vector<double> t64;
        if (int rc = std_load_dust_emission(root, c.dust_emission_lib, c.lam, d.qpah, d.umin, t64, err)) return rc;
        nq = (long long)d.qpah.size();
        nu = (long long)d.umin.size();
        tab.assign(t64.begin(), t64.end());
    } else {
        const std::string dir = root + "/dust_dl07/";
        std::ifstream mf(dir + "manifest.json");
        if (!mf) { err = "dust emission data missing under " + dir; return ST_DATA_MISSING; }
        const std::string text((std::istreambuf_iterator<char>(mf)), std::istreambuf_iterator<char>());
        long long nsf = 0;
        if (!manifest_int(text, "nqpah", nq) || !manifest_int(text, "numin", nu) || !manifest_int(text, "nspec", nsf) ||
            nsf != c.nspec || nq < 2 || nu < 2) {
            err = "dust emission data under " + dir + " does not match the context's grid";
            return ST_DATA_MISSING;
        }
        tab.resize((size_t)ns * nq * 2 * nu);
        std::ifstream tf(dir + "dustem.f32", std::ios::binary);
        if (!read_f64(dir + "qpah.f64", d.qpah, (size_t)nq) || !read_f64(dir + "umin.f64", d.umin, (size_t)nu) || !tf ||
            !tf.read(reinterpret_cast<char *>(tab.data()), (std::streamsize)(sizeof(float) * tab.size()))) {
            err = "dust emission data under " + dir + " is incomplete";
            return ST_DATA_MISSING;
        }
    }
    std::vector<float> cnu((size_t)ns, 0.f);
    for (int i = 0; i + 1 < ns; ++i) {
        const double wt = 0.5 * std::fabs(C_LIGHT / c.lam[i + 1] - C_LIGHT / c.lam[i]);
        cnu[i] += (float)wt;
        cnu[i + 1] += (float)wt;
    }
    cudaError_t e;
    if ((e = d.tab.reserve(tab.size())) != cudaSuccess || (e = d.cnu.reserve(cnu.size())) != cudaSuccess ||
        (e = cudaMemcpy(d.tab.p, tab.data(), sizeof(float) * tab.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(d.cnu.p, cnu.data(), sizeof(float) * cnu.size(), cudaMemcpyHostToDevice)) != cudaSuccess) {
        err = std::string("dust emission upload: ") + cudaGetErrorString(e);
        d.release();
        return ST_DATA_MISSING;
    }
    d.nqpah = (int)nq;
    d.numin = (int)nu;
    d.ready = true;
    return 0;
}

// The AGN torus templates from the data root's agn_torus dataset (the reference reads its torus library at setup;
// here the synthetic stand-in), on the context's wavelength grid.
int agn_load(Context &c, std::string &err) {
    if (c.agn.ready) return 0;
    AgnTorus &a = c.agn;
    const std::string root = data_root();
    std::vector<float> tab;
    if (datalib_available(root, "agn_torus", "clumpy")) {
        // the standard format's agn_torus/clumpy library, interpolated onto the grid
        std::vector<double> t64;
        if (int rc = std_load_agn(root, c.lam, a.tau, t64, err)) return rc;
        tab.assign(t64.begin(), t64.end());
    } else {
        const std::string dir = root + "/agn_torus/";
        std::ifstream mf(dir + "manifest.json");
        if (!mf) { err = "AGN torus data missing under " + dir; return ST_DATA_MISSING; }
        const std::string text((std::istreambuf_iterator<char>(mf)), std::istreambuf_iterator<char>());
        long long ntau = 0, ns = 0;
        if (!manifest_int(text, "ntau", ntau) || !manifest_int(text, "nspec", ns) || ns != c.nspec || ntau < 2) {
            err = "AGN torus data under " + dir + " does not match the context's grid";
            return ST_DATA_MISSING;
        }
        tab.resize((size_t)ntau * ns);
        std::ifstream tf(dir + "agnspec.f32", std::ios::binary);
        if (!read_f64(dir + "tau.f64", a.tau, (size_t)ntau) || !tf ||
            !tf.read(reinterpret_cast<char *>(tab.data()), (std::streamsize)(sizeof(float) * tab.size()))) {
            err = "AGN torus data under " + dir + " is incomplete";
            return ST_DATA_MISSING;
        }
    }
    cudaError_t e;
    if ((e = a.spec.reserve(tab.size())) != cudaSuccess ||
        (e = cudaMemcpy(a.spec.p, tab.data(), sizeof(float) * tab.size(), cudaMemcpyHostToDevice)) != cudaSuccess) {
        err = std::string("AGN torus upload: ") + cudaGetErrorString(e);
        a.release();
        return ST_DATA_MISSING;
    }
    a.ready = true;
    return 0;
}

int context_load_filters(Context &c, const std::string &name, std::string &err) {
    int nb = 0;
    std::vector<double> bands, centers;
    const std::string root = data_root();
    if (datalib_available(root, "filters", name)) {
        // the standard format's filters/<name> library: curves resampled onto the grid, pivot wavelengths
        std::vector<std::string> names;
        if (int rc = std_load_filters(root, name, c.lam, bands, centers, names, err)) return rc;
        nb = (int)centers.size();
        if (nb < 1) { err = "filter library " + name + " has no filters"; return 324; }
    } else {
        if (name == "gauss20") nb = 20;
        else if (name == "gauss40") nb = 40;
        else { err = "unknown filter library " + name; return 324; }
        const std::string dir = root + "/synthetic/";
        if (!read_f64(dir + "filters_" + std::to_string(nb) + ".f64", bands, (size_t)nb * c.nspec) ||
            !read_f64(dir + "filters_" + std::to_string(nb) + "_center.f64", centers, nb)) {
            err = "filter library " + name + " missing under " + dir;
            return 324;
        }
    }
    c.bands.swap(bands);
    c.band_center.swap(centers);
    c.nbands = nb;
    c.filter_set = name;
    c.mag_mask.clear();
    // The band matrix of the split-K product (prepare_batch_grid src/spectra/opensps_batch_photometry.f90:375-392):
    // C(j, b) = band(j, b) (wtl(j - 1) + wtl(j)), wtl(j) = |lambda(j + 1) - lambda(j)| / 2, formed in FP64.
    const int ns = c.nspec;
    std::vector<double> wtl(ns, 0.0);
    for (int j = 0; j + 1 < ns; ++j) wtl[j] = 0.5 * std::fabs(c.lam[j + 1] - c.lam[j]);
    std::vector<double> cm((size_t)nb * ns, 0.0);
    int j0 = ns, j1 = -1;
    for (int b = 0; b < nb; ++b) {
        const double *bd = c.bands.data() + (size_t)b * ns;
        int ilo = ns, ihi = -1;
        for (int j = 0; j < ns; ++j)
            if (bd[j] != 0.0) { ilo = std::min(ilo, j); ihi = std::max(ihi, j); }
        // trapezoid intervals touching the support: j = ilo - 1 .. ihi (0-based), last interval ns - 2
        int jlo = std::max(0, ilo - 1), jhi = std::min(ns - 2, ihi);
        if (ilo > ihi) continue;
        for (int j = 0; j < ns; ++j) {
            double cw = 0.0;
            if (j >= jlo && j <= jhi) cw += wtl[j];
            if (j - 1 >= jlo && j - 1 <= jhi) cw += wtl[j - 1];
            cm[(size_t)b * ns + j] = bd[j] * cw;
        }
        // pixels whose weight can be nonzero: jlo .. jhi + 1
        j0 = std::min(j0, jlo);
        j1 = std::max(j1, jhi + 1);
    }
    if (j1 < j0) { j0 = 0; j1 = -1; }
    // the band GEMM's B operand: rows = bands (padded to npad), columns = pixels j0 .. j0 + 64 nkb - 1, bf16 hi + lo;
    // each pixel's 1 / lambda (the observed-frame spectrum's division by the wavelength) folded in here, in FP64, so
    // that the kernel's operand builders do not multiply by it
    const int npad = band_gemm_npad(nb);
    if (npad > 256) { err = "more than 256 bands"; return ST_BAD_ARG; }
    const int nkb = (j1 - j0 + 1 + 63) / 64, kpad = 64 * nkb;
    std::vector<uint16_t> hi((size_t)npad * std::max(kpad, 64), 0), lo(hi.size(), 0);
    for (int b = 0; b < nb; ++b)
        for (int k = 0; k < kpad; ++k) {
            const int j = j0 + k;
            if (j >= ns) break;
            const double inv_l = c.lam[j] > 2.2250738585072014e-308 ? 1.0 / c.lam[j] : 0.0;
            const float f = (float)(cm[(size_t)b * ns + j] * inv_l);
            const uint16_t h = f32_to_bf16_bits(f);
            hi[(size_t)b * kpad + k] = h;
            lo[(size_t)b * kpad + k] = f32_to_bf16_bits(f - bf16_bits_to_f32(h));
        }
    cudaError_t e;
    if ((e = upload(c.d_cb_hi, reinterpret_cast<const __nv_bfloat16 *>(hi.data()), hi.size())) != cudaSuccess ||
        (e = upload(c.d_cb_lo, reinterpret_cast<const __nv_bfloat16 *>(lo.data()), lo.size())) != cudaSuccess ||
        (e = encode_tmap_2d_bf16(&c.tm_cb_hi, c.d_cb_hi.p, std::max(kpad, 64), npad, 64, npad)) != cudaSuccess ||
        (e = encode_tmap_2d_bf16(&c.tm_cb_lo, c.d_cb_lo.p, std::max(kpad, 64), npad, 64, npad)) != cudaSuccess) {
        err = std::string("band matrix upload failed: ") + cudaGetErrorString(e);
        return ST_BAD_ARG;
    }
    // the same matrix by band for the reverse pass: each band's nonzero pixel range as a dense row, and per chunk of 32
    // pixels from j0 the first and last band reaching it
    std::vector<float> bc;
    std::vector<double> bc64;
    std::vector<int4> bmeta(nb);
    for (int b = 0; b < nb; ++b) {
        int lo = ns, hi = -1;
        for (int j = 0; j < ns; ++j)
            if (cm[(size_t)b * ns + j] != 0.0) { lo = std::min(lo, j); hi = std::max(hi, j); }
        bmeta[b] = make_int4(lo, hi, (int)bc.size(), 0);
        for (int j = lo; j <= hi; ++j) {
            bc.push_back((float)cm[(size_t)b * ns + j]);
            bc64.push_back(cm[(size_t)b * ns + j]);
        }
    }
    const int nchunk = std::max(1, (j1 - j0 + 1 + 31) / 32);
    std::vector<int2> bchunk(nchunk, make_int2(1, 0));
    for (int k = 0; k < nchunk; ++k) {
        const int a0 = j0 + 32 * k, a1 = a0 + 31;
        for (int b = 0; b < nb; ++b) {
            if (bmeta[b].y < a0 || bmeta[b].x > a1 || bmeta[b].y < bmeta[b].x) continue;
            if (bchunk[k].x > bchunk[k].y) bchunk[k] = make_int2(b, b);
            else bchunk[k].y = b;
        }
    }
    if (bc.empty()) { bc.push_back(0.f); bc64.push_back(0.0); }
    if (bmeta.empty()) bmeta.push_back(make_int4(ns, -1, 0, 0));
    if ((e = upload(c.d_bc, bc.data(), bc.size())) != cudaSuccess ||
        (e = upload(c.d_bmeta, bmeta.data(), bmeta.size())) != cudaSuccess ||
        (e = upload(c.d_bc64, bc64.data(), bc64.size())) != cudaSuccess ||
        (e = upload(c.d_bchunk, bchunk.data(), bchunk.size())) != cudaSuccess) {
        err = std::string("band matrix upload failed: ") + cudaGetErrorString(e);
        return ST_BAD_ARG;
    }
    c.band_j0 = j0;
    c.band_j1 = j1;
    c.band_nkb = nkb;
    c.band_npad = npad;
    return 0;
}

// The CLOUDY grid of the setup's isochrone set, when the data root has one: the continuum tables (nodust, dust), the
// nebular ages, the ionizing photon rate of each of their SSPs (nebular_kernels step 1, opensps_csp_batch.f90:2662-2720:
// the frequency trapezoid of L_nu / nu over pixels 1 .. whlylim, times L_sun / h) and per nebular age its CLOUDY age
// interval (batch_nebular_indices :1651-1686). Called from the grid setup once the basis, the pixels below 912 A and
// the line ages are known.
int nebular_load(Context &c, std::string &err) {
    c.neb.release();
    const std::string root = data_root();
    const int ns = c.nspec;
    std::vector<double> tab[2];
    for (int d = 0; d < 2; ++d) {
        const std::string name = c.isoc + (d == 0 ? "_nodust" : "_dust");
        if (!datalib_available(root, "nebular", name)) continue;
        std::vector<double> lz, la, lu;
        if (int rc = std_load_nebular(root, name, c.lam, lz, la, lu, tab[d], err)) return rc;
        if (!c.neb.logz.empty() && (lz != c.neb.logz || la != c.neb.lage || lu != c.neb.logu)) {
            err = "nebular/" + name + ": its axes differ from nebular/" + c.isoc + "_nodust";
            return ST_DATA_MISSING;
        }
        c.neb.logz = lz; c.neb.lage = la; c.neb.logu = lu;
        c.neb.have[d] = true;
    }
    if (!c.neb.have[0] && !c.neb.have[1]) return 0;
    c.nt_neb = std::max(0, std::min(find_interval0(c.log_age.data(), c.nt, c.neb.lage[NEB_NAGE - 1]) + 1, c.nt));
    // per pixel the offset: the grid's largest log2 value there, rounded up (the device tables hold the rest, <= 0)
    const double L2 = 3.321928094887362;   // log2(10)
    std::vector<float> off(ns, 0.f);
    for (int j = 0; j < ns; ++j) {
        double mx = -1e300;
        for (int d = 0; d < 2; ++d)
            if (c.neb.have[d])
                for (size_t k = 0; k < (size_t)NEB_NZ * NEB_NAGE * NEB_NU; ++k) mx = std::max(mx, tab[d][k * ns + j] * L2);
        off[j] = (float)std::ceil(mx);
    }
    cudaError_t e = cudaSuccess;
    for (int d = 0; d < 2 && e == cudaSuccess; ++d) {
        if (!c.neb.have[d]) continue;
        std::vector<float> t((size_t)ns * NEB_NZ * NEB_NAGE * NEB_NU);
        for (int z = 0; z < NEB_NZ; ++z)
            for (int u = 0; u < NEB_NU; ++u)
                for (int a = 0; a < NEB_NAGE; ++a) {
                    const double *src = tab[d].data() + (size_t)ns * (z + NEB_NZ * (a + (size_t)NEB_NAGE * u));
                    float *dst = t.data() + (size_t)ns * (a + NEB_NAGE * (u + (size_t)NEB_NU * z));
                    for (int j = 0; j < ns; ++j) dst[j] = (float)(src[j] * L2 - (double)off[j]);
                }
        e = upload(c.neb.tab[d], t.data(), t.size());
    }
    if (e == cudaSuccess) e = upload(c.neb.off, off.data(), off.size());
    // the ionizing photon rate of each nebular age's SSPs (q0(t, z), metallicity fastest); nu = c / lambda
    const int nn = std::max(c.nt_neb, 1);
    std::vector<double> q0((size_t)nn * c.nz, 0.0);
    if (c.whlylim >= 2)
        for (int z = 0; z < c.nz; ++z)
            for (int t = 0; t < c.nt_neb; ++t) {
                const double *b = c.ssp.data() + (size_t)ns * (t + (size_t)c.nt * z);
                double s = 0.0;
                for (int i = 0; i + 1 < c.whlylim && i + 1 < ns; ++i) {
                    const double n0 = C_LIGHT / c.lam[i], n1 = C_LIGHT / c.lam[i + 1];
                    s += 0.5 * std::fabs(n1 - n0) * (b[i] / n0 + b[i + 1] / n1);
                }
                q0[(size_t)t * c.nz + z] = s / 6.62607015e-27 * 3.828e33;
            }
    // as FP32 scaled by a power of two (their largest in [0.5, 1)): the per-model weights' sums run in FP32
    double qmax = 0.0;
    for (double v : q0) qmax = std::max(qmax, v);
    int qe = 0;
    if (qmax > 0.0) std::frexp(qmax, &qe);
    c.neb.q0_exp = qe;
    std::vector<float> q0s(q0.size());
    for (size_t i = 0; i < q0.size(); ++i) q0s[i] = (float)std::ldexp(q0[i], -qe);
    if (e == cudaSuccess) e = upload(c.neb.q0, q0s.data(), q0s.size());
    // per nebular age its CLOUDY interval: get_grid_indices_weights (opensps_gas.f90:394-412) on the log ages
    c.neb.ia.assign(nn, 0);
    c.neb.wa.assign(nn, 0.0);
    for (int t = 0; t < c.nt_neb; ++t) {
        int k = find_interval0(c.neb.lage.data(), NEB_NAGE, c.log_age[t]);
        k = std::max(0, std::min(k, NEB_NAGE - 2));
        c.neb.ia[t] = k;
        const double w = (c.log_age[t] - c.neb.lage[k]) / (c.neb.lage[k + 1] - c.neb.lage[k]);
        c.neb.wa[t] = std::max(0.0, std::min(w, 1.0));
    }
    if (e != cudaSuccess) {
        err = std::string("nebular grid: ") + cudaGetErrorString(e);
        c.neb.release();
        return ST_DATA_MISSING;
    }
    return 0;
}

// The nebular ages as runs for the continuum kernel: consecutive ages of one CLOUDY interval, on one side of itesc
// (young below it), whose weights wa step uniformly (ages below the grid's first age, wa clamped to 0, form a run of
// step 0). Each run: (first age, count | young << 16, wa of its last age, the step). Built once per itesc.
int nebular_runs(Context &c, int itesc, std::string &err) {
    static_assert(NEB_NAGE <= NEB_RUN_HEAD, "the runs' head holds one int per CLOUDY age");
    if (c.neb.runs_itesc == itesc && c.neb.runs.p) return 0;
    const int nn = c.nt_neb;
    std::vector<int> head(NEB_RUN_HEAD, 0);
    std::vector<int4> runs;
    auto fbits = [](double x) { float f = (float)x; int b; std::memcpy(&b, &f, 4); return b; };
    int t = 0;
    for (int k = 0; k < NEB_NAGE - 1; ++k) {
        head[k] = (int)runs.size();
        while (t < nn && c.neb.ia[t] == k) {
            // a run from t: as long as the interval, the side of itesc and the step hold
            int u = t + 1;
            const bool young = t < itesc;
            double step = 0.0;
            if (u < nn && c.neb.ia[u] == k && (u < itesc) == young) {
                step = c.neb.wa[u] - c.neb.wa[t];
                ++u;
                while (u < nn && c.neb.ia[u] == k && (u < itesc) == young &&
                       std::fabs((c.neb.wa[u] - c.neb.wa[u - 1]) - step) <= 1e-9)
                    ++u;
            }
            const int cnt = u - t;
            const double d = cnt > 1 ? (c.neb.wa[u - 1] - c.neb.wa[t]) / (cnt - 1) : 0.0;
            runs.push_back(make_int4(t, cnt | (young ? 1 << 16 : 0), fbits(c.neb.wa[u - 1]), fbits(d)));
            t = u;
        }
    }
    head[NEB_NAGE - 1] = (int)runs.size();
    if (t != nn || (int)runs.size() > NEB_MAX_RUNS) {
        err = "nebular continuum: the nebular ages do not form runs by interval";
        return ST_UNSUPPORTED;
    }
    c.neb.h_runs.assign(head.begin(), head.end());
    for (const int4 &r : runs) c.neb.h_runs.insert(c.neb.h_runs.end(), {r.x, r.y, r.z, r.w});
    cudaError_t e = c.neb.runs.reserve(c.neb.h_runs.size());
    if (e == cudaSuccess)
        e = cudaMemcpy(c.neb.runs.p, c.neb.h_runs.data(), sizeof(int) * c.neb.h_runs.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        err = std::string("nebular continuum runs: ") + cudaGetErrorString(e);
        c.neb.runs_itesc = -1;
        return ST_DATA_MISSING;
    }
    c.neb.runs_itesc = itesc;
    c.neb.nrun = (int)runs.size();
    return 0;
}

int context_setup(Context &c, const char *isoc, const char *spec, const char *dust, std::string &err) {
    const std::string iso = isoc && *isoc ? isoc : "synthetic", sp = spec ? spec : "";
    const std::string root = data_root();
    if (root.empty()) {
        err = "OPENSPS_DATA_HOME is not set";
        return ST_DATA_MISSING;
    }
    if (data_format_from_env() == DF_BAD) {
        err = "OPENSPS_DATA_FORMAT must be legacy, standard or auto";
        return ST_BAD_ARG;
    }
    // the dust emission library of the batches' add_dust_emission (DL07 unless named)
    const std::string dn = dust ? dust : "";
    c.dust_emission_lib = (dn == "DL07" || dn == "THEMIS") ? dn : "DL07";
    c.dustem.release();
    c.agn.release();
    c.neb.release();
    c.isoc = iso;
    if (datalib_available(root, "ssp", iso)) {
        // an SSP library in the standard format (kind ssp, the isochrone name: read_bpass_standard); its spectra
        // are the basis, so spec_type is not read
        SspLibrary L;
        if (int rc = std_load_ssp(root, iso, L, err)) return rc;
        c.nspec = L.nspec; c.nt = L.nt; c.nz = L.nz; c.nline = L.nline; c.zsol = L.zsol;
        c.lam.swap(L.lam); c.log_age.swap(L.log_age); c.zlegend.swap(L.zlegend); c.ssp.swap(L.spec);
        c.mass.swap(L.mass); c.lbol.swap(L.lbol); c.line_lambda.swap(L.line_lambda); c.line_lum.swap(L.line_lum);
        return context_setup_grid(c, err);
    }
    if (iso != "synthetic" || !(sp.empty() || sp == "synthetic")) {
        err = "library ssp/" + iso + " not found under " + root +
              "/libraries (standard format) and only the synthetic library is in the package's own layout";
        return ST_DATA_MISSING;
    }
    const std::string dir = root + "/synthetic/";
    std::ifstream mf(dir + "manifest.json");
    if (!mf) {
        err = "no synthetic library under " + dir;
        return ST_DATA_MISSING;
    }
    std::stringstream ss;
    ss << mf.rdbuf();
    const std::string man = ss.str();
    long long ns = 0, nt = 0, nz = 0, nl = 0;
    if (!manifest_int(man, "nspec", ns) || !manifest_int(man, "ntfull", nt) || !manifest_int(man, "nz", nz) ||
        !manifest_int(man, "nline", nl)) {
        err = "bad manifest " + dir + "manifest.json";
        return ST_DATA_MISSING;
    }
    manifest_double(man, "zsol", c.zsol);
    c.nspec = (int)ns; c.nt = (int)nt; c.nz = (int)nz; c.nline = (int)nl;
    if (!read_f64(dir + "lambda.f64", c.lam, ns) || !read_f64(dir + "log_age.f64", c.log_age, nt) ||
        !read_f64(dir + "zlegend.f64", c.zlegend, nz) || !read_f64(dir + "ssp_spec.f64", c.ssp, ns * nt * nz) ||
        !read_f64(dir + "ssp_mass.f64", c.mass, nt * nz) || !read_f64(dir + "ssp_lbol.f64", c.lbol, nt * nz) ||
        !read_f64(dir + "line_lambda.f64", c.line_lambda, nl) ||
        !read_f64(dir + "line_lum.f64", c.line_lum, nl * nt * nz)) {
        err = "missing or short array under " + dir;
        return ST_DATA_MISSING;
    }
    return context_setup_grid(c, err);
}

// The rest of the setup from the loaded basis (grid checks, device tables, filters).
int context_setup_grid(Context &c, std::string &err) {
    const int ns = c.nspec;
    // the nebular ranges: whlylim = find_interval(lambda, 912 A) (opensps_initialization.f90:866), and the ages with
    // nebular emission (the nebular grid's age range, opensps_csp_batch.f90:1644-1645: here the ages up to the last
    // one with line luminosity)
    c.whlylim = std::max(find_interval0(c.lam.data(), ns, 912.0) + 1, 0);
    c.nt_neb = 0;
    for (int z = 0; z < c.nz; ++z)
        for (int t = 0; t < c.nt; ++t)
            for (int l = 0; l < c.nline; ++l)
                if (c.line_lum[l + (size_t)c.nline * (t + (size_t)c.nt * z)] != 0.0) c.nt_neb = std::max(c.nt_neb, t + 1);
    // with a CLOUDY grid (nebular/<isoc>_nodust or _dust of a standard-format root) its ages set the nebular ages:
    // nt_neb = find_interval(time_full, nebem_age(NEBNAGE)) (batch_nebular_indices :1643-1644)
    if (int rc = nebular_load(c, err)) return rc;
    c.llin.resize(c.lbol.size());
    for (size_t i = 0; i < c.lbol.size(); ++i) c.llin[i] = std::pow(10.0, c.lbol[i]);
    // the observed-frame resampling and the smoothing taps take the grid as log-uniform: check it
    c.dlnl = (std::log(c.lam[ns - 1]) - std::log(c.lam[0])) / (double)(ns - 1);
    for (int j = 0; j < ns; ++j) {
        const double dev = std::log(c.lam[j]) - std::log(c.lam[0]) - j * c.dlnl;
        if (std::fabs(dev) > 1e-9 * c.dlnl) {
            err = "the wavelength grid is not log-uniform";
            return ST_UNSUPPORTED;
        }
    }

    cudaError_t e = cudaGetDevice(&c.device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c.num_sms, cudaDevAttrMultiProcessorCount, c.device);
    int major = 0, minor = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, c.device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, c.device);
    if (e != cudaSuccess) {
        err = std::string("no CUDA device: ") + cudaGetErrorString(e);
        return ST_DATA_MISSING;
    }
    if (major != 10 || minor != 3) {
        err = "this library is built for sm_103a (GB300); device is sm_" + std::to_string(major) + std::to_string(minor);
        return ST_UNSUPPORTED;
    }
    if ((!c.stream && (e = cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking)) != cudaSuccess) ||
        (!c.side && (e = cudaStreamCreateWithFlags(&c.side, cudaStreamNonBlocking)) != cudaSuccess) ||
        (!c.side2 && (e = cudaStreamCreateWithFlags(&c.side2, cudaStreamNonBlocking)) != cudaSuccess) ||
        (!c.side3 && (e = cudaStreamCreateWithFlags(&c.side3, cudaStreamNonBlocking)) != cudaSuccess) ||
        (!c.side4 && (e = cudaStreamCreateWithFlags(&c.side4, cudaStreamNonBlocking)) != cudaSuccess) ||
        (!c.ev_cot && (e = cudaEventCreateWithFlags(&c.ev_cot, cudaEventDisableTiming)) != cudaSuccess) ||
        (!c.ev_w0 && (e = cudaEventCreateWithFlags(&c.ev_w0, cudaEventDisableTiming)) != cudaSuccess) ||
        (!c.ev_w1 && (e = cudaEventCreateWithFlags(&c.ev_w1, cudaEventDisableTiming)) != cudaSuccess) ||
        (!c.ev_contract && (e = cudaEventCreateWithFlags(&c.ev_contract, cudaEventDisableTiming)) != cudaSuccess) ||
        (!c.ev_fork && (e = cudaEventCreateWithFlags(&c.ev_fork, cudaEventDisableTiming)) != cudaSuccess) ||
        (!c.ev_params && (e = cudaEventCreateWithFlags(&c.ev_params, cudaEventDisableTiming)) != cudaSuccess) ||
        (!c.ev_sums && (e = cudaEventCreateWithFlags(&c.ev_sums, cudaEventDisableTiming)) != cudaSuccess)) {
        err = std::string("stream: ") + cudaGetErrorString(e);
        return ST_DATA_MISSING;
    }

    // per-pixel table
    c.jtop = 0;
    for (int j = 0; j < ns; ++j)
        if (c.lam[j] < 1215.67) c.jtop = j + 1;
    std::vector<float> wl(ns), igm_a((size_t)std::max(c.jtop, 1) * 6, 0.f);
    for (int j = 0; j < ns; ++j) wl[j] = c.lam[j] > 2.2250738585072014e-308 ? (float)(1.0 / c.lam[j]) : 0.f;
    for (int j = 0; j < c.jtop; ++j) {
        double a[6];
        igm_pixel_terms(c.lam[j], a);
        for (int k = 0; k < 6; ++k) igm_a[(size_t)j * 6 + k] = (float)a[k];
    }
    c.igm_a = igm_a;
    std::vector<double> igm_a64((size_t)std::max(c.jtop, 1) * 6, 0.0);
    for (int j = 0; j < c.jtop; ++j) igm_pixel_terms(c.lam[j], igm_a64.data() + (size_t)j * 6);
    std::vector<double> lnlam(ns);
    for (int j = 0; j < ns; ++j) lnlam[j] = std::log(c.lam[j]);
    c.lzv.resize(c.nz);
    for (int z = 0; z < c.nz; ++z) c.lzv[z] = std::log10(c.zlegend[z] / c.zsol);
    cosmology_table(c.h0, c.om0, c.ol0, c.zt, c.dl);
    std::vector<double> ages(c.log_age);   // log10 of the grid's ages, then the ages (yr)
    for (int t = 0; t < c.nt; ++t) ages.push_back(std::pow(10.0, c.log_age[t]));
    if ((e = upload(c.d_wl, wl.data(), wl.size())) != cudaSuccess ||
        (e = upload(c.d_igm_a, igm_a.data(), igm_a.size())) != cudaSuccess ||
        (e = upload(c.d_igm_a64, igm_a64.data(), igm_a64.size())) != cudaSuccess ||
        (e = upload(c.d_lam, c.lam.data(), c.lam.size())) != cudaSuccess ||
        (e = upload(c.d_lnlam, lnlam.data(), lnlam.size())) != cudaSuccess ||
        (e = upload(c.d_mass, c.mass.data(), c.mass.size())) != cudaSuccess ||
        (e = upload(c.d_llin, c.llin.data(), c.llin.size())) != cudaSuccess ||
        (e = upload(c.d_logage, ages.data(), ages.size())) != cudaSuccess ||
        (e = upload(c.d_lz, c.lzv.data(), c.lzv.size())) != cudaSuccess ||
        (e = upload(c.d_lbol, c.lbol.data(), c.lbol.size())) != cudaSuccess ||
        (e = upload(c.d_zt, c.zt.data(), c.zt.size())) != cudaSuccess ||
        (e = upload(c.d_dl, c.dl.data(), c.dl.size())) != cudaSuccess ||
        (e = c.d_status.reserve(4)) != cudaSuccess) {
        err = std::string("device upload failed: ") + cudaGetErrorString(e);
        return ST_DATA_MISSING;
    }
    // the nebular ages' ionizing pixels (their escaping fraction is added per model when frac_obrun > 0)
    c.d_ion.release();
    if (c.nt_neb > 0 && c.whlylim > 0) {
        const int whl = c.whlylim, ntn = c.nt_neb;
        std::vector<float> ion((size_t)c.nz * ntn * whl);
        for (int z = 0; z < c.nz; ++z)
            for (int t = 0; t < ntn; ++t)
                for (int i = 0; i < whl; ++i)
                    ion[((size_t)z * ntn + t) * whl + i] = (float)c.ssp[i + (size_t)ns * (t + (size_t)c.nt * z)];
        if ((e = upload(c.d_ion, ion.data(), ion.size())) != cudaSuccess) {
            err = std::string("device upload failed: ") + cudaGetErrorString(e);
            return ST_DATA_MISSING;
        }
    }
    c.d_pix.release();   // rebuilt by the next batch (smoothing range)
    c.pix_key[0] = -1e300;
    int st = context_load_filters(c, c.filter_set, err);
    if (st != 0) return st;
    for (auto &kv : c.basis_cache) { kv.second->release(); delete kv.second; }
    c.basis_cache.clear();
    c.eml_nnz = -1;
    // the no-allocation magnitudes' modules and scratch address on this device (so that its calls allocate nothing)
    if ((e = noalloc_prepare(c.device)) != cudaSuccess) {
        err = std::string("loading the no-allocation entry point's modules: ") + cudaGetErrorString(e);
        return ST_DATA_MISSING;
    }
    c.sm_range[0] = 0.0;
    c.sm_range[1] = -1.0;
    c.line_thr = -1.0;
    c.is_setup = true;
    return 0;
}

}  // namespace sps
