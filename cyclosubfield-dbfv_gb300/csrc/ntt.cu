// Lazy radix-2/3 group NTTs along dimension 2 or 3 of a ring-element tensor.
//
// The reference applies, per cyclic factor and per stage, Cooley-Tukey butterflies whose twiddle
// products are Barrett multiplications and whose sums stay unreduced; full reduction passes are
// inserted only where a data-independent worst-case bound says the next stage could overflow
// (cyclosubfield-dbfv/src/hal/ntt.rs:301-537, plan level :581-657). Because that schedule does
// not depend on the data, the host simulates it once per plan and stores a *stage program*
// (radix, geometry, reduce-before, twiddle-1 skip permission, fused final reduction/scaling)
// next to the twiddle constants in device memory. The kernel executes the program over a tile
// held in shared memory: a dimension-3 line (one CTA per line), or a block of dimension-2
// columns (one CTA per column block). Each butterfly performs exactly the reference's integer
// formula, so outputs are bit-identical; stages are not algebraically merged.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "ntt_tile.cuh"

namespace {

// ---------------------------------------------------------------- host-side constants
int64_t h_mul_mod(int64_t a, int64_t b, int64_t q) { return (int64_t)(((i128)a * (i128)b) % (i128)q); }
int64_t h_pow_mod(int64_t b, uint64_t e, int64_t q) {
    int64_t r = 1;
    b %= q;
    while (e) {
        if (e & 1) r = h_mul_mod(r, b, q);
        b = h_mul_mod(b, b, q);
        e >>= 1;
    }
    return r;
}
bool is_pow2(uint64_t x) { return x && !(x & (x - 1)); }
int64_t h_find_root(int64_t q, uint64_t n) {
    uint64_t p = is_pow2(n) ? 2 : 3;
    for (int64_t c = 2;; c++) {
        int64_t root = h_pow_mod(c, (uint64_t)((q - 1) / (int64_t)n), q);
        if (h_pow_mod(root, n / p, q) != 1) return root;
    }
}
/// BarrettMul::new (src/hal/ntt.rs:134-144): centred z, u = round(-z 2^64 / n).
void h_barrett(int64_t value, int64_t n, int64_t* z_out, int64_t* u_out) {
    int64_t z = value % n;
    if (2 * (i128)z > n) z -= n;
    else if (2 * (i128)z < -n) z += n;
    i128 a = -((i128)z << 64), b = n;
    i128 u = a >= 0 ? (a + b / 2) / b : -((-a + b / 2) / b);
    *z_out = z;
    *u_out = (int64_t)u;
}

/// Moduli and lazy bounds of the limb products (barrett_mul, mont_mul).
const int64_t LIMB_MOD_MAX = (int64_t)1 << 57;
const u128 LIMB_BOUND_MAX = (u128)8301034833169298227ull;  // 0.9 x 2^63

struct HostPlan {
    DevPlanHeader h;
    std::vector<int64_t> tw;  // pairs
    std::vector<BarrettLimbs> limbs;  // of each pair, for n < 2^57
    void push(int64_t value) {
        int64_t z, u;
        h_barrett(value, h.n, &z, &u);
        if (h.n < LIMB_MOD_MAX) limbs.push_back(barrett_limbs(z, u, h.n));
        tw.push_back(z);
        tw.push_back(u);
    }
    int32_t next_tw() const { return (int32_t)(tw.size() / 2); }
};

const u128 I64MAX = (u128)INT64_MAX;

}  // namespace

struct hc_ntt_plan_s {
    void* dev;        // DevPlanHeader + twiddles
    int64_t n;
    int32_t len;
    int32_t ntw;      // twiddle pairs
    int32_t counts[4];  // stages forward and inverse, passes forward and inverse
    int32_t shape;    // HC_SHAPE_*: factorisation with a specialised kernel
    bool fixed;       // the schedule is the shape's compiled-in one and the limb products are exact
    size_t bytes;
};

// ---------------------------------------------------------------- device kernel
namespace {

#ifndef HC_NTT_MIN_BLOCKS
#define HC_NTT_MIN_BLOCKS 3  // resident CTAs per SM the register allocation must allow
#endif

/// mode 0: forward (reduced), 1: inverse, 2: forward unreduced + Montgomery multiplication by `mul`.
/// dim 3: tile = line (i, j, k), element e at l = e.  dim 2: tile = (i, j, column block),
/// element (e, v) at k = e, l = cb * V + v.
__global__ void __launch_bounds__(256, HC_NTT_MIN_BLOCKS) ntt_tile_kernel(KView t, PlanPtrs plans, int dim, int mode, KView mul,
                                                       KMods mods, int logv, int ntile2, int use_smem) {
    grid_wait();
    extern __shared__ __align__(16) int64_t smem[];
    const int V = 1 << logv;
    const int len = dim == 3 ? (int)t.n3 : (int)t.n2;
    int64_t tile = blockIdx.x;
    int64_t i, j, k = 0, cb = 0;
    if (dim == 3) {
        k = tile % t.n2;
        int64_t r = tile / t.n2;
        j = r % t.n1;
        i = r / t.n1;
    } else {
        cb = tile % ntile2;
        int64_t r = tile / ntile2;
        j = r % t.n1;
        i = r / t.n1;
    }
    const DevPlanHeader* P = plans.p[j];
    // the plan's twiddle constants are staged in shared memory, behind the tile
    int64_t* tws = smem + (use_smem ? (size_t)len * V : 0);
    stage_twiddles(P, tws);
    TileIO io;
    io.g = reinterpret_cast<int64_t*>(t.p) + i * t.s0 + j * t.s1 + (dim == 3 ? k * t.s2 : cb * V);
    io.ge = dim == 3 ? 1 : t.s2;
    io.ncol = dim == 3 ? 1 : t.n3 - cb * V;
    io.mulp = nullptr, io.me = io.mv = 0, io.mn = io.mi = 0;
    if (mode & 2) {
        io.mulp = kat<int64_t>(mul, i, j, dim == 3 ? k : 0, dim == 3 ? 0 : cb * V);
        io.me = dim == 3 ? (mul.b3 ? 0 : 1) : mul.s2;
        io.mv = dim == 3 ? 0 : (mul.b3 ? 0 : 1);
        io.mn = mods.n[j], io.mi = mods.ninv[j];
    }
    tile_run(P, tws, smem, len, logv, use_smem, mode, io);
}

}  // namespace

// ---------------------------------------------------------------- plan construction
namespace hc {

// the specialised kernels (ntt_line3072.cu, ntt_line12288.cu, ntt_col.cu); mode as ntt_tile_kernel's, 3:
// inverse + Montgomery multiplication; fix: every plan is fixed
hc_status launch_ntt_line3072(hc_context ctx, int mode, bool fix, const KView& t, const PlanPtrs& pp, const KView& mul,
                              const KMods& mods, int64_t tiles);
hc_status launch_ntt_line12288(hc_context ctx, int mode, bool fix, const KView& t, const PlanPtrs& pp, const KView& mul,
                               const KMods& mods, int64_t tiles);
hc_status launch_ntt_col(hc_context ctx, int shape, int mode, bool fix, const KView& t, const PlanPtrs& pp,
                         const KView& mul, const KMods& mods, int64_t tiles, int ncb, const KView& src);

/// Builds the stage programs and twiddle tables of CpuNTTPlan::new (src/hal/ntt.rs:561-566,
/// LazyFactorNTT::new :216-281) and simulates the bound tracking of `apply` (:581-657) and of
/// the factor transforms (:301-537).
hc_status build_plan(hc_context ctx, const hc_modulus* m, const size_t* shape, size_t k, hc_ntt_plan* out) {
    (void)ctx;  // plans live in device memory of the current device, shared by its contexts
    const int64_t n = m->n;
    if (n <= 1 || n % 2 == 0 || n >= ((int64_t)1 << 62)) return fail(HC_ERR_ARG, "NTT modulus must be odd and < 2^62");
    HostPlan hp;
    std::memset(&hp.h, 0, sizeof(hp.h));
    hp.h.n = n;
    std::vector<size_t> factors;
    size_t len = 1;
    for (size_t i = 0; i < k; i++) {
        len *= shape[i];
        if (shape[i] > 1) factors.push_back(shape[i]);
    }
    if (len > ((size_t)1 << 30)) return fail(HC_ERR_UNSUPPORTED, "NTT length too large");
    hp.h.len = (int32_t)len;
    int64_t z, u;
    h_barrett(1, n, &z, &u);
    hp.h.one_z = z, hp.h.one_u = u;
    int64_t inv_len = h_pow_mod((int64_t)(len % (size_t)n), (uint64_t)(n - 2), n);
    h_barrett(inv_len, n, &z, &u);
    hp.h.invlen_z = z, hp.h.invlen_u = u;
    if (n < LIMB_MOD_MAX) hp.h.invlen = barrett_limbs(z, u, n);
    u = hp.h.one_u;
    bool limbs = false;  // the limb products are exact for this modulus and schedule

    if (n < LIMB_MOD_MAX) {
        // u = -2^k for the constant of 1: the reductions are shifts (barrett_red)
        int kk = 0;
        while (kk < 31 && u != -((int64_t)1 << kk)) kk++;
        limbs = kk >= 1 && kk < 31;
        BarrettMod& bm = hp.h.mod;
        bm.n0 = (int32_t)lo32(n), bm.nn0 = (int32_t)lo32(-n), bm.nn1 = bal_hi(-n);
        bm.red_shift = 32 - kk, bm.red_add = kk >= 1 ? (int32_t)(((int64_t)1 << (31 - kk)) - 1) : 0;
    }
    // a reduction by such a constant leaves |x - round(x / 2^(64 - k)) n| <= 2^(63 - k) + (2^k + 1)
    // (2^(64 - k) - n); the largest operand of a product with that in place of n
    const auto after_red = [&]() -> u128 {
        const int lg = 32 + hp.h.mod.red_shift;  // n is near 2^lg
        const u128 top = (u128)1 << lg, d = top > (u128)n ? top - (u128)n : (u128)n - top;
        return (top >> 1) + (((u128)1 << (64 - lg)) + 1) * d;
    };
    u128 fmax = 2 * (u128)n, imax = 2 * (u128)n, flimb = 2 * (u128)n, ilimb = 2 * (u128)n;
    u128 fbound = 2 * (u128)n, ibound = 2 * (u128)n;
    size_t suffix = 1;
    for (size_t f : factors) suffix *= f;
    for (size_t fi = 0; fi < factors.size(); fi++) {
        const size_t flen = factors[fi];
        suffix /= flen;
        const bool last_factor = fi + 1 == factors.size();
        const bool r2 = is_pow2(flen);
        if (!r2) {
            size_t l = flen;
            while (l > 1) {
                if (l % 3) return fail(HC_ERR_ARG, "NTT length must be a power of 2 or a power of 3");
                l /= 3;
            }
        }
        if ((n - 1) % (int64_t)flen) return fail(HC_ERR_ARG, "modulus doesn't support roots of unity of this order");
        if (r2 && 2 * (u128)n > I64MAX) return fail(HC_ERR_ARG, "modulus too large for lazy radix-2 butterflies");
        if (!r2 && 3 * (u128)n > I64MAX) return fail(HC_ERR_ARG, "modulus too large for lazy radix-3 butterflies");
        const int radix = r2 ? 2 : 3;
        int64_t root = h_find_root(n, flen);
        int64_t inv_root = h_pow_mod(root, flen - 1, n);
        // twiddles per stage, in the residue-tree order of src/hal/ntt.rs:226-232 / :250-270
        std::vector<std::vector<int64_t>> fw, iv;
        std::vector<size_t> exps{0};
        int64_t zeta = 0, zeta2 = 0;
        if (!r2) {
            zeta = h_pow_mod(root, flen / 3, n);
            zeta2 = h_mul_mod(zeta, zeta, n);
        }
        while (exps.size() < flen) {
            std::vector<int64_t> f1, i1;
            for (size_t e : exps) {
                if (r2) {
                    f1.push_back(h_pow_mod(root, e / 2, n));
                    i1.push_back(h_pow_mod(inv_root, e / 2, n));
                } else {
                    int64_t v = h_pow_mod(root, e / 3, n), v2 = h_mul_mod(v, v, n);
                    f1.push_back(v);
                    f1.push_back(h_mul_mod(zeta, v, n));
                    f1.push_back(h_mul_mod(zeta2, v, n));
                    f1.push_back(v2);
                    f1.push_back(h_mul_mod(zeta, v2, n));
                    f1.push_back(h_mul_mod(zeta2, v2, n));
                    int64_t vi = h_pow_mod(inv_root, e / 3, n);
                    i1.push_back(vi);
                    i1.push_back(h_mul_mod(vi, vi, n));
                }
            }
            fw.push_back(f1);
            iv.push_back(i1);
            std::vector<size_t> next;
            for (size_t e : exps)
                for (int c = 0; c < radix; c++) next.push_back(e / radix + c * (flen / radix));
            exps.swap(next);
        }
        const size_t nst = fw.size();
        int32_t zeta_off = 0;
        if (!r2) {
            zeta_off = hp.next_tw();
            hp.push(zeta);
            hp.push(zeta2);
        }
        // forward program (src/hal/ntt.rs:312-353, :355-411)
        const int fstart = hp.h.nfwd, istart = hp.h.ninv;
        size_t stage_len = flen;
        for (size_t s = 0; s < nst; s++) {
            if (hp.h.nfwd >= HC_MAX_STAGES) return fail(HC_ERR_UNSUPPORTED, "too many NTT stages");
            DevStage& st = hp.h.fwd[hp.h.nfwd++];
            st.radix = radix;
            st.stride = (int32_t)suffix;
            st.flen = (int32_t)flen;
            st.stage_len = (int32_t)stage_len;
            st.tw_off = hp.next_tw();
            for (int64_t v : fw[s]) hp.push(v);
            st.last = last_factor && s + 1 == nst;
            st.span = (int32_t)((stage_len / radix) * suffix);
            st.div_span = make_fastdiv((uint32_t)st.span);
            st.div_nblocks = make_fastdiv((uint32_t)(flen / stage_len));
            const u128 grow = r2 ? (u128)n : 2 * (u128)n;
            if (fbound + grow > I64MAX) {
                st.reduce_before = 1;
                fbound = (u128)n;
                flimb = after_red();
            }
            st.skip_ok = (u128)radix * fbound <= I64MAX;
            // the unreduced bound is tracked; a fused final reduction only affects the returned
            // bound of the very last stage, which nothing reads
            fbound = st.skip_ok ? (u128)radix * fbound : fbound + grow;
            flimb = st.skip_ok ? (u128)radix * flimb : flimb + grow;
            fmax = std::max(fmax, flimb);  // operand of the next stage or of the fused product
            stage_len /= radix;
        }
        // inverse program (src/hal/ntt.rs:438-478, :480-533): stages in reverse order
        for (size_t si = nst; si-- > 0;) {
            if (hp.h.ninv >= HC_MAX_STAGES) return fail(HC_ERR_UNSUPPORTED, "too many NTT stages");
            DevStage& st = hp.h.inv[hp.h.ninv++];
            st.radix = radix;
            st.stride = (int32_t)suffix;
            st.flen = (int32_t)flen;
            size_t sl = flen;
            for (size_t q = 0; q < si; q++) sl /= radix;
            st.stage_len = (int32_t)sl;
            st.tw_off = hp.next_tw();
            for (int64_t v : iv[si]) hp.push(v);
            st.zeta_off = zeta_off;
            st.last = last_factor && si == 0;
            st.span = (int32_t)((sl / radix) * suffix);
            st.div_span = make_fastdiv((uint32_t)st.span);
            st.div_nblocks = make_fastdiv((uint32_t)(flen / sl));
            if ((u128)radix * ibound > I64MAX) {
                st.reduce_before = 1;
                ibound = (u128)n;
                ilimb = after_red();
            }
            ibound = st.last ? (u128)n : (u128)radix * ibound;
            ilimb = (u128)radix * ilimb;  // operands of this stage's products
            imax = std::max(imax, ilimb);
        }
        // passes: radix-2 stages in register groups of up to three, radix-3 stages one by one
        auto add_pass = [&](bool fwd, int kind, int k, int first, int span, int glen, int nb) {
            int32_t& cnt = fwd ? hp.h.nfpass : hp.h.nipass;
            DevPass& ps = (fwd ? hp.h.fpass : hp.h.ipass)[cnt++];
            ps.kind = kind, ps.k = k, ps.first = first, ps.span = span, ps.glen = glen, ps.nb = nb;
            ps.div_span = make_fastdiv((uint32_t)(span > 0 ? span : 1));
            ps.div_nb = make_fastdiv((uint32_t)(nb > 0 ? nb : 1));
        };
        const int S = (int)suffix, F = (int)flen, NST = (int)nst;
        for (int c = 0; c < NST;) {
            if (!r2) {
                add_pass(true, 0, 1, fstart + c, 0, 0, 0);
                c++;
                continue;
            }
            int k = std::min(3, NST - c);
            int L = F >> c;  // stage length at the pass's first stage
            add_pass(true, 1, k, fstart + c, (L >> k) * S, L * S, F / L);
            c += k;
        }
        for (int c = 0; c < NST;) {
            if (!r2) {
                add_pass(false, 0, 1, istart + c, 0, 0, 0);
                c++;
                continue;
            }
            int k = std::min(3, NST - c);
            int Lp = 2 << c;  // stage length of the first processed stage (si = nst - 1 - c)
            int Llast = Lp << (k - 1);
            add_pass(false, 1, k, istart + c, (Lp / 2) * S, Llast * S, F / Llast);
            c += k;
        }
    }
    hp.h.ntw = hp.next_tw();
    const size_t tw_bytes = hp.tw.size() * sizeof(int64_t);
    size_t bytes = sizeof(DevPlanHeader) + tw_bytes + hp.limbs.size() * sizeof(BarrettLimbs);
    limbs = limbs && fmax <= LIMB_BOUND_MAX && imax <= LIMB_BOUND_MAX;
    int shape_id = HC_SHAPE_GENERIC;
    if (factors == std::vector<size_t>{2, 3, 8, 64}) shape_id = HC_SHAPE_L3072;
    else if (factors == std::vector<size_t>{3, 64, 64}) shape_id = HC_SHAPE_L12288;
    else if (factors == std::vector<size_t>{4, 3}) shape_id = HC_SHAPE_C12;
    else if (factors == std::vector<size_t>{4}) shape_id = HC_SHAPE_C4;
    {
        SchedMasks m{0u, 0u, 0u, 0u, 0u};
        for (int i = 0; i < hp.h.nfwd; i++) {
            m.fred |= (uint32_t)(hp.h.fwd[i].reduce_before != 0) << i;
            m.fskip |= (uint32_t)(hp.h.fwd[i].skip_ok != 0) << i;
            m.flast |= (uint32_t)(hp.h.fwd[i].last != 0) << i;
        }
        for (int i = 0; i < hp.h.ninv; i++) {
            m.ired |= (uint32_t)(hp.h.inv[i].reduce_before != 0) << i;
            m.ilast |= (uint32_t)(hp.h.inv[i].last != 0) << i;
        }
        bool laid = shape_id != HC_SHAPE_GENERIC;  // the table's offsets are the compiled-in ones
        if (laid) {
            const TableLayout t = table_layout(shape_id);
            laid = t.words == hp.next_tw();
            for (int i = 0; i < hp.h.nfwd; i++) laid = laid && hp.h.fwd[i].tw_off == t.fwd[i];
            for (int i = 0; i < hp.h.ninv; i++)
                laid = laid && hp.h.inv[i].tw_off == t.inv[i] && (hp.h.inv[i].radix == 2 || hp.h.inv[i].zeta_off == t.zeta[i]);
        }
        for (int lg : {56, 57}) {
            const SchedMasks f = fixed_masks(shape_id, lg);
            if (limbs && laid && m.fred == f.fred && m.fskip == f.fskip && m.flast == f.flast && m.ired == f.ired &&
                m.ilast == f.ilast)
                hp.h.cls = lg;
        }
    }
    std::vector<char> blob(bytes);
    std::memcpy(blob.data(), &hp.h, sizeof(DevPlanHeader));
    if (!hp.tw.empty()) std::memcpy(blob.data() + sizeof(DevPlanHeader), hp.tw.data(), tw_bytes);
    if (!hp.limbs.empty())
        std::memcpy(blob.data() + sizeof(DevPlanHeader) + tw_bytes, hp.limbs.data(), bytes - sizeof(DevPlanHeader) - tw_bytes);
    void* dev = nullptr;
    count_alloc();
    if (cudaMalloc(&dev, bytes) != cudaSuccess) return fail(HC_ERR_OOM, "cannot allocate NTT plan");
    hc_status st = cuda_check(cudaMemcpy(dev, blob.data(), bytes, cudaMemcpyHostToDevice), "plan upload");
    if (st != HC_OK) {
        cudaFree(dev);
        return st;
    }
    auto* plan = new hc_ntt_plan_s();
    plan->dev = dev;
    plan->shape = shape_id;
    plan->fixed = hp.h.cls != 0;
    plan->n = n;
    plan->len = (int32_t)len;
    plan->ntw = hp.h.ntw;
    plan->counts[0] = hp.h.nfwd, plan->counts[1] = hp.h.ninv, plan->counts[2] = hp.h.nfpass, plan->counts[3] = hp.h.nipass;
    plan->bytes = bytes;
    *out = plan;
    return HC_OK;
}

hc_status destroy_plan(hc_ntt_plan p) {
    if (!p) return HC_OK;
    cudaFree(p->dev);
    delete p;
    return HC_OK;
}

int64_t plan_modulus(hc_ntt_plan p) { return p->n; }
int32_t plan_len(hc_ntt_plan p) { return p->len; }
const void* plan_device(hc_ntt_plan p) { return p->dev; }
int32_t plan_ntw(hc_ntt_plan p) { return p->ntw; }
void plan_counts(hc_ntt_plan p, int32_t counts[4]) { std::copy(p->counts, p->counts + 4, counts); }
int32_t plan_shape(hc_ntt_plan p) { return p->shape | (p->fixed ? 0x100 : 0); }
/// Launches the tile kernel for one HAL NTT call (mode 0 ntt, 1 intt, 2 ntt_mul).
/// Whether launch_ntt runs a call on the specialised column kernel, the one form that can read a
/// separate source (launch_ntt's `src`).
bool ntt_column_path(const hc_ntt_plan* plans, size_t nplans, int dim) {
    if (dim != 2 || nplans == 0 || !plans[0]) return false;
    const int shape = plans[0]->shape;
    for (size_t j = 0; j < nplans; j++)
        if (!plans[j] || plans[j]->shape != shape) return false;
    return shape == HC_SHAPE_C12 || shape == HC_SHAPE_C4;
}

/// Whether launch_ntt can run a call with its multipliers as a table of limbs (mode 6): the specialised
/// kernels over fixed plans.
bool ntt_limb_path(const hc_ntt_plan* plans, size_t nplans, int dim) {
    if (nplans == 0 || !plans[0]) return false;
    const int shape = plans[0]->shape;
    for (size_t j = 0; j < nplans; j++)
        if (!plans[j] || plans[j]->shape != shape || !plans[j]->fixed) return false;
    return dim == 2 ? shape == HC_SHAPE_C12 || shape == HC_SHAPE_C4 : shape == HC_SHAPE_L3072 || shape == HC_SHAPE_L12288;
}

/// mode 6: the forward transform times the limb table mul.p (BarrettLimbs elements, strides in them);
/// only where ntt_limb_path holds.
hc_status launch_ntt(hc_context ctx, const KView& t, const hc_ntt_plan* plans, size_t nplans, int dim, int mode,
                     const KView& mul, const KMods& mods, const KView* src) {
    if (mode == 6 && !ntt_limb_path(plans, nplans, dim)) return fail(HC_ERR_UNSUPPORTED, "limb multipliers of a general NTT");
    if (src && !ntt_column_path(plans, nplans, dim)) return fail(HC_ERR_UNSUPPORTED, "out-of-place NTT form");
    if ((int64_t)nplans != t.n1) return fail(HC_ERR_SHAPE, "one NTT plan per RNS row required");
    if (nplans > HC_MAX_MODS) return fail(HC_ERR_UNSUPPORTED, "too many RNS rows in one call");
    const int64_t len = dim == 3 ? t.n3 : t.n2;
    PlanPtrs pp;
    int32_t max_tw = 0;
    for (size_t j = 0; j < nplans; j++) {
        if (!plans[j]) return fail(HC_ERR_ARG, "null NTT plan");
        if (plans[j]->len != len) return fail(HC_ERR_SHAPE, "NTT plan length does not match the transformed dimension");
        pp.p[j] = reinterpret_cast<const DevPlanHeader*>(plans[j]->dev);
        max_tw = std::max(max_tw, plans[j]->ntw);
    }
    if (t.n0 == 0 || t.n1 == 0 || t.n2 == 0 || t.n3 == 0) return HC_OK;
    int shape = plans[0]->shape;
    for (size_t j = 1; j < nplans; j++)
        if (plans[j]->shape != shape) shape = HC_SHAPE_GENERIC;
    bool fix = true;
    for (size_t j = 0; j < nplans; j++) fix = fix && plans[j]->fixed;
    if (mode == 2) {
        // the limb product of the caller's multipliers wants their moduli below 2^57 (they need not be the plans') and
        // reads some of them again after its first stores, so they may not lie in t (MontAny)
        for (size_t j = 0; j < nplans; j++) fix = fix && mods.n[j] < LIMB_MOD_MAX;
        const int64_t lt = (t.n0 - 1) * t.s0 + (t.n1 - 1) * t.s1 + (t.n2 - 1) * t.s2 + t.n3 - 1;
        const int64_t lm = (t.n0 - 1) * mul.s0 + (t.n1 - 1) * mul.s1 + (t.n2 - 1) * mul.s2 + (mul.b3 ? 0 : t.n3 - 1);
        fix = fix && (mul.p > t.p + 8 * lt || t.p > mul.p + 8 * lm);
    }
    if (dim == 3 && (shape == HC_SHAPE_L3072 || shape == HC_SHAPE_L12288)) {
        const int64_t tiles = t.n0 * t.n1 * t.n2;
        if (tiles <= 0x7fffffff)
            return shape == HC_SHAPE_L3072 ? launch_ntt_line3072(ctx, mode, fix, t, pp, mul, mods, tiles)
                                           : launch_ntt_line12288(ctx, mode, fix, t, pp, mul, mods, tiles);
    }
    if (dim == 2 && (shape == HC_SHAPE_C12 || shape == HC_SHAPE_C4)) {
        const int64_t ncb = (t.n3 + HC_COL_THREADS - 1) / HC_COL_THREADS;
        const int64_t tiles = t.n0 * t.n1 * ncb;
        if (tiles <= 0x7fffffff)
            return launch_ntt_col(ctx, shape, mode, fix, t, pp, mul, mods, tiles, (int)ncb, src ? *src : KView());
    }
    if (src || mode == 6) return fail(HC_ERR_UNSUPPORTED, "specialised NTT form");
    int V = 1, logv = 0;
    int64_t ntile2 = 1;
    if (dim == 2) {
        // as many dimension-3 columns per tile as fit into 48 KB of shared memory (<= 64)
        V = 64;
        while (V > 1 && (len * V * 8 > 49152 || V / 2 >= t.n3)) V /= 2;
        while ((1 << logv) < V) logv++;
        ntile2 = (t.n3 + V - 1) / V;
    }
    const size_t tw_bytes = (size_t)max_tw * 16;
    size_t smem = (size_t)len * V * 8 + tw_bytes;
    int use_smem = 1;
    size_t maxs = max_smem_optin(ctx);
    if (smem > maxs) {
        if (dim == 2) return fail(HC_ERR_UNSUPPORTED, "dimension-2 NTT length too large");
        use_smem = 0;
        smem = tw_bytes;
        if (smem > maxs) return fail(HC_ERR_UNSUPPORTED, "NTT twiddle table too large");
    }
    if (smem > 49152) {
        cudaError_t e = cudaFuncSetAttribute(ntt_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return cuda_check(e, "ntt smem attribute");
    }
    int64_t tiles = dim == 3 ? t.n0 * t.n1 * t.n2 : t.n0 * t.n1 * ntile2;
    if (tiles > 0x7fffffff) return fail(HC_ERR_UNSUPPORTED, "too many NTT tiles in one call");
    // about 24 elements (three groups of eight) per thread, 64..256 threads
    int64_t threads = ((len * V / 24) + 31) / 32 * 32;
    threads = threads < 64 ? 64 : (threads > 256 ? 256 : threads);
    hc::launch_kernel(ntt_tile_kernel, (unsigned)tiles, (unsigned)threads, smem, stream_of(ctx), t, pp, dim, mode, mul, mods, logv,
                                                                    (int)ntile2, use_smem);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "ntt kernel launch");
}

}  // namespace hc
