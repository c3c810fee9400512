// se2p_tc.cu -- Gaussian spread and gather on the tensor cores (FP64 form).
//
// The spread of a tile of sources is a contraction: with X_s[i], Y_s[j] the
// one-dimensional Gaussian factors of source s (zero outside its P + 1
// nodes), the grid patch around the tile receives
//     H_c[i][j] += sum_s (c_s X_s[i]) Y_s[j],
// a matrix product over the tile's sources.  Tensor cores multiply 16-bit
// floats, so both factors are written as fixed-point numbers of 64 bits and
// cut into base-256 digits -128 .. 127, each exact in FP16.  A product of two
// digits is below 2^14 and the FP32 accumulator holds integers exactly up to
// 2^24, so the sums of all digit pairs (p, q) with p + q = l, "level l", are
// exact integers for up to kTcMaxK sources, and the patch is
// sum_l level_l 256^-l: an integer result, independent of the order of the
// sources.  Levels below the last are dropped (2^-56 of the largest |c| per
// source for 7 levels), rounded once per node where the sums
// join the int64 grids at scale 2^S, the same grids k_spread_fix fills.
#include "se2p_internal.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <climits>

namespace se2p {

// ---------------------------------------------------------------------------
// Points -> stencil factors, tiles, items
// ---------------------------------------------------------------------------

// Fixed point.  FP64 instructions issue at 1/70 of the integer rate here, so the
// Gaussian factors are fractions of 2^64 formed with integer products.

// a b / 2^64, within about one unit: the low halves' product is left out and the
// added 1 makes up for it and for the two dropped fractions on average.
__device__ __forceinline__ unsigned long long mulhi_apx(unsigned long long a, unsigned long long b)
{
    const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32);
    const uint32_t bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
    return (unsigned long long)ah * bh + __umulhi(ah, bl) + (unsigned long long)__umulhi(al, bh) + 1;
}

// 2^(-j/256) 2^64, rounded (j = 0: 2^64 - 1).
__constant__ unsigned long long c_exp2_tab[256] = {
    0xffffffffffffffffull, 0xff4ecb59511ec8a5ull, 0xfe9e115c7b8f884cull, 0xfdedd1b496a89f35ull,
    0xfd3e0c0cf486c175ull, 0xfc8ec01121e447bbull, 0xfbdfed6ce5f09c49ull, 0xfb3193cc4227c3f4ull,
    0xfa83b2db722a033aull, 0xf9d64a46eb939f35ull, 0xf92959bb5dd4ba74ull, 0xf87ce0e5b2094d9cull,
    0xf7d0df730ad13bb9ull, 0xf7255510c4288239ull, 0xf67a416c733f846eull, 0xf5cfa433e6537290ull,
    0xf5257d152486cc2cull, 0xf47bcbbe6db9fddfull, 0xf3d28fde3a641a5bull, 0xf329c9233b6bae9cull,
    0xf281773c59ffb13aull, 0xf1d999d8b7708cc1ull, 0xf13230a7ad094509ull, 0xf08b3b58cbe8b76aull,
    0xefe4b99bdcdaf5cbull, 0xef3eab20e032bc6bull, 0xee990f980da3025bull, 0xedf3e6b1d418a491ull,
    0xed4f301ed9942b84ull, 0xecaaeb8ffb03ab41ull, 0xec0718b64c1cbddcull, 0xeb63b74317369840ull,
    0xeac0c6e7dd24392full, 0xea1e4756550eb27bull, 0xe97c38406c4f8c57ull, 0xe8da9958464b42abull,
    0xe8396a503c4bdc68ull, 0xe798aadadd5b9cbfull, 0xe6f85aaaee1fce22ull, 0xe658797368b3a717ull,
    0xe5b906e77c8348a8ull, 0xe51a02ba8e26d681ull, 0xe47b6ca0373da88dull, 0xe3dd444c46499619ull,
    0xe33f8972be8a5a51ull, 0xe2a23bc7d7d91226ull, 0xe2055afffe83d369ull, 0xe168e6cfd3295d23ull,
    0xe0ccdeec2a94e111ull, 0xe031430a0d99e627ull, 0xdf9612deb8f04420ull, 0xdefb4e1f9d1037f2ull,
    0xde60f4825e0e9124ull, 0xddc705bcd378f7f0ull, 0xdd2d818508324c20ull, 0xdc9467913a4f1c92ull,
    0xdbfbb797daf23755ull, 0xdb63714f8e295255ull, 0xdacb946f2ac9cc72ull, 0xda3420adba4d8704ull,
    0xd99d15c278afd7b6ull, 0xd9067364d44a929cull, 0xd870394c6db32c84ull, 0xd7da67311797f56aull,
    0xd744fccad69d6af4ull, 0xd6aff9d1e13ba2feull, 0xd61b5dfe9f9bce07ull, 0xd5872909ab75d18aull,
    0xd4f35aabcfedfa1full, 0xd45ff29e0972c561ull, 0xd3ccf099859ac379ull, 0xd33a5457a3029054ull,
    0xd2a81d91f12ae45aull, 0xd2164c023056bcabull, 0xd184df6251699ac6ull, 0xd0f3d76c75c5db8dull,
    0xd06333daef2b2595ull, 0xcfd2f4683f94eeb5ull, 0xcf4318cf191918c1ull, 0xceb3a0ca5dc6a55dull,
    0xce248c151f8480e4ull, 0xcd95da6a9ff06445ull, 0xcd078b86503dcdd2ull, 0xcc799f23d11510e5ull,
    0xcbec14fef2727c5dull, 0xcb5eecd3b38597c9ull, 0xcad2265e4290774eull, 0xca45c15afcc72624ull,
    0xc9b9bd866e2f27a3ull, 0xc92e1a9d517f0eccull, 0xc8a2d85c8ffe2c45ull, 0xc817f681416452b2ull,
    0xc78d74c8abb9b15dull, 0xc70352f04336c51eull, 0xc67990b5aa245f79ull, 0xc5f02dd6b0bbc3d9ull,
    0xc5672a115506daddull, 0xc4de8523c2c07baaull, 0xc4563ecc5334cb33ull, 0xc3ce56c98d21b15dull,
    0xc346ccda24976407ull, 0xc2bfa0bcfad907c9ull, 0xc238d2311e3d6673ull, 0xc1b260f5ca0fbb33ull,
    0xc12c4cca66709456ull, 0xc0a6956e8836ca8dull, 0xc0213aa1f0d08db0ull, 0xbf9c3c248e2486f8ull,
    0xbf1799b67a731083ull, 0xbe935317fc378238ull, 0xbe0f6809860993e2ull, 0xbd8bd84bb67ed483ull,
    0xbd08a39f580c36bfull, 0xbc85c9c560e7b269ull, 0xbc034a7ef2e9fb0dull, 0xbb81258d5b704b6full,
    0xbaff5ab2133e45fbull, 0xba7de9aebe5fea09ull, 0xb9fcd2452c0b9debull, 0xb97c143756844dbfull,
    0xb8fbaf4762fb9ee9ull, 0xb87ba337a1743834ull, 0xb7fbefca8ca41e7cull, 0xb77c94c2c9d725e9ull,
    0xb6fd91e328d17791ull, 0xb67ee6eea3b22b8full, 0xb60093a85ed5f76cull, 0xb58297d3a8b9f0d2ull,
    0xb504f333f9de6484ull, 0xb487a58cf4a9c180ull, 0xb40aaea2654b9841ull, 0xb38e0e38419fae18ull,
    0xb311c412a9112489ull, 0xb295cff5e47db4a4ull, 0xb21a31a66618fe3bull, 0xb19ee8e8c94feb09ull,
    0xb123f581d2ac2590ull, 0xb0a957366fb7a3c9ull, 0xb02f0dcbb6e04584ull, 0xafb51906e75b8661ull,
    0xaf3b78ad690a4375ull, 0xaec22c84cc5c9465ull, 0xae493452ca35b80eull, 0xadd08fdd43d01491ull,
    0xad583eea42a14ac6ull, 0xace0413ff83e5d04ull, 0xac6896a4be3fe929ull, 0xabf13edf162675e9ull,
    0xab7a39b5a93ed337ull, 0xab0386ef48868de1ull, 0xaa8d2652ec907629ull, 0xaa1717a7b5693979ull,
    0xa9a15ab4ea7c0ef8ull, 0xa92bef41fa77771bull, 0xa8b6d5167b320e09ull, 0xa8420bfa298f70d1ull,
    0xa7cd93b4e965356aull, 0xa7596c0ec55ff55bull, 0xa6e594cfeee86b1eull, 0xa6720dc0be08a20cull,
    0xa5fed6a9b15138eaull, 0xa58bef536dbeb6eeull, 0xa5195786be9ef339ull, 0xa4a70f0c95768ec5ull,
    0xa43515ae09e6809eull, 0xa3c36b345991b47cull, 0xa3520f68e802bb93ull, 0xa2e102153e918f9eull,
    0xa27043030c496819ull, 0xa1ffd1fc25cea188ull, 0xa18faeca8544b6e4ull, 0xa11fd9384a344cf7ull,
    0xa0b0510fb9714fc2ull, 0xa041161b3d0121beull, 0x9fd228256400dd06ull, 0x9f6386f8e28ba651ull,
    0x9ef5326091a111aeull, 0x9e872a276f0b98ffull, 0x9e196e189d472420ull, 0x9dabfdff6367a2aaull,
    0x9d3ed9a72cffb751ull, 0x9cd200db8a0774cbull, 0x9c6573682ec32c2dull, 0x9bf93118f3aa4cc1ull,
    0x9b8d39b9d54e5539ull, 0x9b218d16f441d63dull, 0x9ab62afc94ff864aull, 0x9a4b13371fd166caull,
    0x99e0459320b7fa65ull, 0x9975c1dd47518c77ull, 0x990b87e266c189aaull, 0x98a1976f7597e996ull,
    0x9837f0518db8a96full, 0x97ce9255ec4357abull, 0x97657d49f17ab08eull, 0x96fcb0fb20ac4ba3ull,
    0x96942d3720185a00ull, 0x962bf1cbb8d97560ull, 0x95c3fe86d6cc7fefull, 0x955c5336887894d5ull,
    0x94f4efa8fef70961ull, 0x948dd3ac8ddb7ed3ull, 0x9426ff0fab1c04b6ull, 0x93c071a0eef94bc1ull,
    0x935a2b2f13e6e92cull, 0x92f42b88f673aa7cull, 0x928e727d9531f9acull, 0x9228ffdc10a051adull,
    0x91c3d373ab11c336ull, 0x915eed13c89689d3ull, 0x90fa4c8beee4b12bull, 0x9095f1abc540ca6bull,
    0x9031dc431466b1dcull, 0x8fce0c21c6726481ull, 0x8f6a8117e6c8e5c4ull, 0x8f073af5a2013520ull,
    0x8ea4398b45cd53c0ull, 0x8e417ca940e35a01ull, 0x8ddf042022e69cd6ull, 0x8d7ccfc09c50e2f8ull,
    0x8d1adf5b7e5ba9e6ull, 0x8cb932c1bae97a95ull, 0x8c57c9c4646f4ddeull, 0x8bf6a434adde0085ull,
    0x8b95c1e3ea8bd6e7ull, 0x8b3522a38e1e1032ull, 0x8ad4c6452c728924ull, 0x8a74ac9a79896e47ull,
    0x8a14d575496efd9aull, 0x89b540a7902557a4ull, 0x8955ee03618e5fddull, 0x88f6dd5af155ac6bull,
    0x88980e8092da8527ull, 0x88398146b919f1d4ull, 0x87db357ff698d792ull, 0x877d2afefd4e256cull,
    0x871f61969e8d1010ull, 0x86c1d919caef5c88ull, 0x8664915b923fba04ull, 0x86078a2f23642a9full,
    0x85aac367cc487b15ull, 0x854e3cd8f9c8c95dull, 0x84f1f656379c1a29ull, 0x8495efb3303efd30ull,
    0x843a28c3acde4046ull, 0x83dea15b9541b132ull, 0x8383594eefb6ee37ull, 0x83285071e0fc4547ull,
    0x82cd8698ac2ba1d7ull, 0x8272fb97b2a5894cull, 0x8218af4373fc25ecull, 0x81bea1708dde6056ull,
    0x8164d1f3bc030773ull, 0x810b40a1d81406d4ull, 0x80b1ed4fd999ab6cull, 0x8058d7d2d5e5f6b1ull,
};

// 2^-y as a fraction of 2^64, y in units of 2^-59: the table method, y = n / 256
// + f, 2^-f = exp(-r), r = f ln 2 < 0.0028, exp(-r) = 1 - r + r^2/2 (1 - h) with
// h = r (1/3 - r/12 + r^2/60) in 40 bits (the next Taylor term is below 2^-60).
__device__ __forceinline__ unsigned long long exp2_neg_fix(unsigned long long y,
                                                           const unsigned long long *tab)
{
    const int n = (int)(y >> 51);
    const unsigned long long f = (y & ((1ull << 51) - 1)) << 5;      // f 2^64, f < 2^-8
    const unsigned long long r = mulhi_apx(f, 0xb17217f7d1cf79acull); // ln 2
    const uint32_t r40 = (uint32_t)(r >> 24);                        // r 2^40
    uint32_t k = 0x15555555u - (uint32_t)(((unsigned long long)r40 * 0x4444444u) >> 40);  // 1/12 - r/60
    k = 0x55555555u - (uint32_t)(((unsigned long long)r40 * k) >> 40);                    // 1/3 - ...
    const unsigned long long h = (unsigned long long)__umulhi(r40, k) << 24;
    const unsigned long long r2 = mulhi_apx(r, r) >> 1;
    const unsigned long long e = 0ull - r + r2 - mulhi_apx(r2, h);   // exp(-r) 2^64 (r >= 1)
    const unsigned long long v = mulhi_apx(tab[n & 255], e);
    const int sh = n >> 8;
    return sh < 64 ? v >> sh : 0;
}

// Per point: the Gaussian factor at the nearest node and the two ratios to the
// nodes beside it, per axis, as fractions of 2^64.  meta: offset of the stencil
// origin within its tile (x, y), and whether the nearest node is P/2 or P/2 + 1.
struct __align__(16) TcPoint {
    unsigned long long ex, qpx, qmx, ey, qpy, qmy;
    int meta, pad[3];
};
static_assert(sizeof(TcPoint) == kTcPointBytes, "record size");

__device__ __forceinline__ int tc_wrap(int i, int M)
{
    i %= M;
    return i < 0 ? i + M : i;
}

// Stencil origin along one axis, and the offset from it in nodes as a fraction
// of 2^64: closest_node's arithmetic wherever x lies within `near` nodes of one (2^-20,
// and more where h is so small that its snap at 1e-13 reaches farther), elsewhere
// products with 1/h in place of its divisions (no decision is near).
__device__ __forceinline__ bool tc_axis(double x, double Lh, double h, double inv_h, double near, int half,
                                        int &m, unsigned long long &u)
{
    const double q = x * inv_h, fl = floor(q);
    const double t = (x + Lh) * inv_h, ft = floor(t);
    const double fr = q - fl, gr = t - ft;
    m = (int)ft - half;
    const double o = xsub(x, xmul(h, fl)) * inv_h;
    // o 2^64 from the bit pattern (2^-20 < o < 1 where it counts)
    const unsigned long long b = (unsigned long long)__double_as_longlong(o);
    u = ((b << 11) | (1ull << 63)) >> (1022 - (int)(b >> 52));
    const double hi = 1.0 - near;
    return fr > near && fr < hi && gr > near && gr < hi && fabs(x) < 1e9 * h;
}

// The factors X[i] = exp(-alpha (u - (i - P/2))^2), u in [0, 1) the offset in
// nodes, follow outward from the node nearest to the point: X[i +- 1] = X[i] q,
// q' = q exp(-2 alpha), with q <= 1 on both sides.
__device__ __forceinline__ void tc_seed(unsigned long long u, unsigned long long al,
                                        const unsigned long long *tab, int &b, unsigned long long &e,
                                        unsigned long long &qp, unsigned long long &qm)
{
    b = (int)(u >> 63);
    const unsigned long long d = b ? 0ull - u : u;   // distance to the nearest node (< 2^63, 1/2 of 2^64)
    e = exp2_neg_fix(mulhi_apx(al, mulhi_apx(d, d)), tab);
    // alpha (1 -+ 2 d)
    const unsigned long long w = min(mulhi_apx(al, d) << 1, al);
    const unsigned long long near = exp2_neg_fix(al - w, tab), far = exp2_neg_fix(al + w, tab);
    // u below the node's cell middle: the point lies above the node
    qp = b ? far : near;
    qm = b ? near : far;
}

// Bound: issue (about 400 integer instructions per point).  With the exponentials,
// divisions and conversions in FP64 it took 310 us for 2^20 points, bound by the FP64 pipe.
__global__ void __launch_bounds__(256) k_tc_points(TcPrepArgs b)
{
    chain_enter();
    const TcPointArgs &a = b.s[blockIdx.y].a;
    __shared__ unsigned long long tab[256];
    tab[threadIdx.x] = c_exp2_tab[threadIdx.x];
    __syncthreads();
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= a.n) return;
    const double2 S = a.p[j];
    int mx, my;
    unsigned long long ux, uy;
    const bool okx = tc_axis(S.x, a.Lhx, a.h, a.inv_h, a.near, a.P / 2, mx, ux);
    const bool oky = tc_axis(S.y, a.Lhy, a.h, a.inv_h, a.near, a.P / 2, my, uy);
    if (!(okx && oky)) {
        double px, py;
        closest_node(S.x, S.y, a.Lhx, a.Lhy, a.h, a.P, mx, my, px, py);
        ux = __double2ull_rn(fmin(fmax(px / a.h, 0.0), 1.0) * 0x1p64);
        uy = __double2ull_rn(fmin(fmax(py / a.h, 0.0), 1.0) * 0x1p64);
    }
    const int cx = tc_wrap(mx, a.Mx), cy = tc_wrap(my, a.My);
    const int tx = cx / a.Tx, ty = cy / a.Ty;
    const int tile = tx * a.nty + ty;
    int bx, by;
    TcPoint r;
    tc_seed(ux, a.al2, tab, bx, r.ex, r.qpx, r.qmx);
    tc_seed(uy, a.al2, tab, by, r.ey, r.qpy, r.qmy);
    r.meta = (cx - tx * a.Tx) | (cy - ty * a.Ty) << 8 | bx << 16 | by << 17;
    r.pad[0] = r.pad[1] = r.pad[2] = 0;
    reinterpret_cast<TcPoint *>(a.fac)[j] = r;
    // (box-sorted points: a warp's lanes mostly share a tile)
    const unsigned act = __activemask();
    const unsigned m = __match_any_sync(act, tile);
    const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
    int base = 0;
    if (lane == lead) base = atomicAdd(&a.count[tile], __popc(m));
    base = __shfl_sync(m, base, lead);
    a.tile[j] = make_int2(tile, base + __popc(m & ((1u << lane) - 1u)));
}

// Exclusive scans of the tiles' counts and of their numbers of items,
// ceil(count / kmax) each: a block scans 1024 tiles and adds up the counts before
// them itself (23 blocks at 2688^2 nodes: 4 us; one block over all of them, 30 us).
__global__ void __launch_bounds__(1024) k_tc_items(TcPrepArgs b)
{
    chain_enter();
    const TcSetArgs &t = b.s[blockIdx.y];
    const int *__restrict__ count = t.a.count;
    const int ntile = t.ntile, kmax = t.kmax;
    if ((int)blockIdx.x * 1024 >= ntile) return;
    // ceil(v / kmax) by a product with ceil(2^32 / kmax), exact for kmax <= 64 and v
    // below 2^25; larger counts divide
    const unsigned inv = 0xffffffffu / (unsigned)kmax + 1;
    auto chunks = [&](int v) {
        const unsigned a = (unsigned)(v + kmax - 1);
        return (int)(v < 1 << 25 ? __umulhi(a, inv) : a / (unsigned)kmax);
    };
    __shared__ int2 warp_tot[32], before[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int base = blockIdx.x * 1024, i = base + tid;
    int2 pre = make_int2(0, 0);
    for (int k = tid; k < base; k += 1024) {
        const int v = count[k];
        pre.x += v;
        pre.y += chunks(v);
    }
    const int v = i < ntile ? count[i] : 0;
    const int2 own = make_int2(v, chunks(v));
    int2 inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(~0u, inc.x, o), y = __shfl_up_sync(~0u, inc.y, o);
        if (lane >= o) {
            inc.x += x;
            inc.y += y;
        }
        pre.x += __shfl_xor_sync(~0u, pre.x, o);
        pre.y += __shfl_xor_sync(~0u, pre.y, o);
    }
    if (lane == 31) {
        warp_tot[wid] = inc;
        before[wid] = pre;
    }
    __syncthreads();
    int2 run = make_int2(inc.x - own.x, inc.y - own.y);
    for (int w = 0; w < 32; w++) {
        run.x += before[w].x + (w < wid ? warp_tot[w].x : 0);
        run.y += before[w].y + (w < wid ? warp_tot[w].y : 0);
    }
    if (i < ntile) {
        t.start[i] = run.x;
        t.istart[i] = run.y;
        if (i == ntile - 1) {
            t.start[ntile] = run.x + own.x;
            *t.nitems = run.y + own.y;
        }
    }
}

// Slot -> sorted point, tile by tile, and the items: a tile's points cut into
// nearly equal runs, items[k] = (tile, first slot, count, 0).  key: the
// points' numbers in the caller's order, by slot (with perm).
__global__ void __launch_bounds__(256) k_tc_list(TcPrepArgs b)
{
    chain_enter();
    const TcSetArgs &w = b.s[blockIdx.y];
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= w.a.n) return;
    const int2 t = w.a.tile[j];
    const int a = w.start[t.x], v = w.start[t.x + 1] - a;
    w.list[a + t.y] = (int)j;
    if (w.perm) w.key[a + t.y] = w.perm[j];
    const int nch = (v + w.kmax - 1) / w.kmax;
    const int c = (int)(((int64_t)t.y * nch + nch - 1) / v);
    const int first = (int)((int64_t)v * c / nch);
    if (c < nch && first == t.y)
        w.items[w.istart[t.x] + c] = make_int4(t.x, a + first, (int)((int64_t)v * (c + 1) / nch) - first, 0);
}

// A tile of more than one item: its slots in the order of the caller's point
// numbers, so that each item holds the same points on every call (the digit
// sums are exact, but each item's patch is rounded to the grid's unit once).
// The other tiles keep the order the atomics gave them.  A block ranks 256
// slots by counting smaller keys, the keys read through shared memory.
// With nbound right-hand sides on the same sources the list serves them all, so it is
// left unwritten only where none of their spreads will read it.
// The ranking grows with the square of a tile's slots: beyond kOrderFrom sources
// k_tc_order_long takes the tiles of more than kOrderLong.
constexpr int kOrderLong = 4096, kOrderFrom = 1 << 16;

__device__ __forceinline__ bool all_off(const unsigned long long *__restrict__ bound, int nbound, int bstride)
{
    if (bound[0] != kFixedOff) return false;
    for (int r = 1; r < nbound; r++)
        if (bound[(int64_t)r * bstride] != kFixedOff) return false;
    return true;
}

__global__ void __launch_bounds__(256) k_tc_order(int64_t n, const int2 *__restrict__ tile,
                                                  const int *__restrict__ start, int kmax, int longest,
                                                  const int *__restrict__ key,
                                                  const int *__restrict__ list,
                                                  int *__restrict__ out,
                                                  const unsigned long long *__restrict__ bound,
                                                  int nbound, int bstride)
{
    chain_enter();
    if (all_off(bound, nbound, bstride)) return;     // crowded: the FP64 spread runs instead
    __shared__ __align__(16) int ks[256];
    __shared__ int range[2];
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (threadIdx.x == 0) {
        range[0] = 0x7fffffff;
        range[1] = 0;
    }
    __syncthreads();
    int a = 0, b = 0, j = 0, mine = 0;
    if (k < n) {
        j = list[k];
        const int t = tile[j].x;
        a = start[t];
        b = start[t + 1];
        if (b - a > longest) {
            b = a;
        } else if (b - a > kmax) {
            mine = key[k];
            atomicMin(&range[0], a);
            atomicMax(&range[1], b);
        } else {
            out[k] = j;
            b = a;
        }
    }
    __syncthreads();
    const int lo = range[0], hi = range[1];
    int r = 0;
    for (int m0 = lo; m0 < hi; m0 += 256) {
        if (m0 + (int)threadIdx.x < hi) ks[threadIdx.x] = key[m0 + threadIdx.x];
        __syncthreads();
        const int e0 = max(a - m0, 0), e1 = min(b - m0, 256);
        if (e0 == 0 && e1 == 256) {
#pragma unroll 8
            for (int e = 0; e < 64; e++) {
                const int4 q = reinterpret_cast<const int4 *>(ks)[e];
                r += (q.x < mine) + (q.y < mine) + (q.z < mine) + (q.w < mine);
            }
        } else {
            for (int e = e0; e < e1; e++) r += ks[e] < mine;
        }
        __syncthreads();
    }
    if (b > a) out[a + r] = j;
}

// Tiles of more than kOrderLong slots (coarse grids, and sources without a density, which
// the bound does not count as crowded), a block each: the keys, which are distinct, fall
// into up to kOrderBins equal intervals between their least and their largest, and
// are ranked within their interval.  tmp: room for the n slots' keys, then for their points.
// Bound: latency of one block's passes over its tile.  Whole k-space calls, ranking by
// squares alone against this: 2^17 sources of one tile, 50 of them with a density, 2.44
// against 0.65 ms, 2^19 27.8 against 2.26; 2^20 uniform sources on 128^2 nodes, P = 4, 11.6
// against 2.33 ms, on 256^2, P = 12, 3.46 against 2.07.  At the line both take the same (one
// tile of 4096: 0.24 ms; of 8192: 0.27 against 0.25).  Its launch is 3 us of every call
// (32,768 boundary points 484 against 487 us), so that up to kOrderFrom sources, 0.44
// against 0.32 ms at most for 2^15, there is none.
constexpr int kOrderThreads = 1024, kOrderLogBins = 13, kOrderBins = 1 << kOrderLogBins;

__global__ void __launch_bounds__(kOrderThreads) k_tc_order_long(int64_t n, int ntile, const int *__restrict__ start,
                                                                 const int *__restrict__ key,
                                                                 const int *__restrict__ list,
                                                                 int *__restrict__ out, int *tmp,
                                                                 const unsigned long long *__restrict__ bound,
                                                                 int nbound, int bstride)
{
    chain_enter();
    if (all_off(bound, nbound, bstride)) return;
    __shared__ int bins[kOrderBins], found[kOrderThreads], warp_tot[kOrderThreads / 32], nfound, klo, khi;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int64_t t0 = blockIdx.x; t0 < ntile; t0 += (int64_t)gridDim.x * kOrderThreads) {
        const int64_t t = t0 + (int64_t)tid * gridDim.x;
        const bool mine = t < ntile && start[t + 1] - start[t] > kOrderLong;
        if (!__syncthreads_or(mine)) continue;
        if (tid == 0) nfound = 0;
        __syncthreads();
        if (mine) found[atomicAdd(&nfound, 1)] = (int)t;
        __syncthreads();
        for (int f = 0; f < nfound; f++) {
            const int first = start[found[f]], end = start[found[f] + 1];
            if (tid == 0) {
                klo = 0x7fffffff;
                khi = 0;
            }
            for (int q = tid; q < kOrderBins; q += kOrderThreads) bins[q] = 0;
            __syncthreads();
            int lo = 0x7fffffff, hi = 0;
            for (int k = first + tid; k < end; k += kOrderThreads) {
                lo = min(lo, key[k]);
                hi = max(hi, key[k]);
            }
            lo = __reduce_min_sync(~0u, lo);
            hi = __reduce_max_sync(~0u, hi);
            if (lane == 0) {
                atomicMin(&klo, lo);
                atomicMax(&khi, hi);
            }
            __syncthreads();
            const int base = klo, sh = max(0, 32 - kOrderLogBins - __clz(khi - klo));   // (hi - lo) >> sh < kOrderBins
            for (int k = first + tid; k < end; k += kOrderThreads) atomicAdd(&bins[(key[k] - base) >> sh], 1);
            __syncthreads();
            // the bins' first places: an exclusive scan, kPer consecutive bins per thread
            constexpr int kPer = kOrderBins / kOrderThreads;
            int c[kPer], sum = 0;
#pragma unroll
            for (int q = 0; q < kPer; q++) sum += c[q] = bins[tid * kPer + q];
            int inc = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int x = __shfl_up_sync(~0u, inc, d);
                if (lane >= d) inc += x;
            }
            if (lane == 31) warp_tot[wid] = inc;
            __syncthreads();
            int run = first + inc - sum;
            for (int w = 0; w < wid; w++) run += warp_tot[w];
#pragma unroll
            for (int q = 0; q < kPer; q++) {
                bins[tid * kPer + q] = run;
                run += c[q];
            }
            __syncthreads();
            for (int k = first + tid; k < end; k += kOrderThreads) {
                const int v = key[k], m = atomicAdd(&bins[(v - base) >> sh], 1);
                tmp[m] = v;
                tmp[n + m] = list[k];
            }
            __syncthreads();
            // (a bin's word is now the end of its interval)
            for (int k = first + tid; k < end; k += kOrderThreads) {
                const int v = tmp[k], q = (v - base) >> sh, a = q ? bins[q - 1] : first, b = bins[q];
                int r = a, m = a;
                for (; m < b && (m & 3); m++) r += tmp[m] < v;
                for (; m + 4 <= b; m += 4) {
                    const int4 w = *reinterpret_cast<const int4 *>(tmp + m);
                    r += (w.x < v) + (w.y < v) + (w.z < v) + (w.w < v);
                }
                for (; m < b; m++) r += tmp[m] < v;
                out[r] = tmp[n + k];
            }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// tcgen05, mbarrier and bulk-copy instructions
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// One poll, of up to 20 us, of the phase of the given parity.
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 20000;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok;
}

__device__ __forceinline__ void tc_give_up(const TcWait &w)
{
    *w.bad = 1;
    *w.err = 1;
    __threadfence_system();
}

// Waits for the phase of the given parity; gives up after w.polls polls (or when another
// thread has), sets the shared abort flag and the error words, and returns false.  What the
// phase guards is then not there: the thread must touch none of it and go to the next of
// its group's barriers, which end with tc_stop for all threads of the group together.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_sh,
                                          const TcWait &w)
{
    for (int i = 0; i < w.polls; i++) {
        if (mbar_poll(bar, parity)) return true;
        if (*abort_sh) return false;
    }
    *abort_sh = 1;
    tc_give_up(w);
    return false;
}

// Barrier of THREADS threads that says whether any of them has seen the abort flag: the
// same answer for all, so that they leave their loops together.
template <int ID, int THREADS>
__device__ __forceinline__ bool tc_stop(volatile int *abort_sh)
{
    uint32_t stop;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\t"
                 "bar.red.or.pred q, %2, %3, p;\n\t"
                 "selp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(stop)
                 : "r"(*abort_sh), "n"(ID), "n"(THREADS)
                 : "memory");
    return stop;
}

__device__ __forceinline__ void tc_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// The end of the issuing thread: everything it issued must have completed before shared
// memory and TMEM are given back, also where its waits have given up.
__device__ __forceinline__ void tc_drain(uint32_t bar, const TcWait &w)
{
    tc_commit(bar);
    for (int i = 0; i < kTcPolls; i++)
        if (mbar_poll(bar, 0)) return;
    tc_give_up(w);
}

__device__ __forceinline__ void fence_async_shared()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// *dst += *src, u64 by u64, as an asynchronous bulk reduction (16-byte units).
__device__ __forceinline__ void bulk_add_u64(void *dst, uint32_t src, int bytes)
{
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.u64 [%0], [%1], %2;" ::"l"(dst),
                 "r"(src), "r"(bytes)
                 : "memory");
}

// D[128 x N] (+)= A[128 x 16] B[16 x N], FP16 operands in shared memory.
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                 "l"(a), "l"(b), "r"(idesc), "r"(acc)
                 : "memory");
}

// Shared-memory matrix descriptor, no swizzle: 8 x 16 B core matrices, lbo and
// sbo their strides in bytes (MN-major: lbo along K, sbo along M / N; K-major:
// lbo along K, sbo along M / N).
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3fff) | (uint64_t)((lbo >> 4) & 0x3fff) << 16 |
           (uint64_t)((sbo >> 4) & 0x3fff) << 32 | (uint64_t)1 << 46;
}

// Instruction descriptor: FP32 accumulator, FP16 operands, M = 128, N.
__device__ __forceinline__ uint32_t tc_idesc(int N, int mn_major)
{
    return 1u << 4 | (mn_major ? 3u << 15 : 0u) | (uint32_t)(N >> 3) << 17 | 8u << 24;
}

__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

// Waits for the loads; the registers pass through so that nothing reads them earlier.
__device__ __forceinline__ void tc_ld_wait8(uint32_t (&r)[8])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7])::"memory");
}

// ---------------------------------------------------------------------------
// Digits
// ---------------------------------------------------------------------------
constexpr int kTcDigits = 7;
// Base-256 digits of four numbers up to 2^63, most significant first, as FP16,
// each number's digits times its sign: adding 128 to every byte but the top one
// carries the digits' signs upward, so the top byte is a digit 0 .. 128 and the
// others less 128 are digits -128 .. 127; 0x6400 | byte is the FP16 number 1024
// + byte.  Digit p's four go to dst + p stride as
// one 8-byte store.
template <int NS>
__device__ __forceinline__ void store_digits(const unsigned long long (&v)[4], __half2 sign, char *dst,
                                             int stride)
{
    uint32_t out[8][2];
    const __half2 off = __hmul2(sign, __float2half2_rn(-1152.0f)), off0 = __hmul2(sign, __float2half2_rn(-1024.0f));
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const unsigned long long a = v[2 * k] + 0x0080808080808080ull;
        const unsigned long long b = v[2 * k + 1] + 0x0080808080808080ull;
#pragma unroll
        for (int w = 0; w < 2; w++) {                // high word, low word
            const uint32_t aw = (uint32_t)(w ? a : a >> 32), bw = (uint32_t)(w ? b : b >> 32);
            const uint32_t z = __byte_perm(aw, bw, 0x7632), y = __byte_perm(aw, bw, 0x5410);
            const uint32_t d[4] = {__byte_perm(z, 0x64646464u, 0x4341), __byte_perm(z, 0x64646464u, 0x4240),
                                   __byte_perm(y, 0x64646464u, 0x4341), __byte_perm(y, 0x64646464u, 0x4240)};
#pragma unroll
            for (int q = 0; q < 4; q++) {            // sign (1024 + byte) - sign (1024 or 1152)
                const __half2 h = __hfma2(*reinterpret_cast<const __half2 *>(&d[q]), sign, w + q ? off : off0);
                out[4 * w + q][k] = *reinterpret_cast<const uint32_t *>(&h);
            }
        }
    }
#pragma unroll
    for (int p = 0; p < NS; p++)
        *reinterpret_cast<uint2 *>(dst + p * stride) = make_uint2(out[p][0], out[p][1]);
}

template <int NS>
__device__ __forceinline__ void store_zero_digits(char *dst, int stride)
{
#pragma unroll
    for (int p = 0; p < NS; p++) *reinterpret_cast<uint2 *>(dst + p * stride) = make_uint2(0, 0);
}

// One side of one axis of a point's factors, as fractions of 2^64, from the
// centre outward into rows i, i + di, .. (n of them) of a window of rows STRIDE
// apart, then zeros up to the window's end.
template <int STRIDE>
__device__ __forceinline__ void tc_factors(unsigned long long e, unsigned long long q,
                                           unsigned long long s, int i, int di, int n, int win,
                                           unsigned long long *out)
{
    unsigned long long *o = out + i * STRIDE;
    const int step = di * STRIDE, left = di > 0 ? win - i - n : i + 1 - n;
    for (int k = 0; k < n; k++) {
        *o = e;
        e = mulhi_apx(e, q);
        q = mulhi_apx(q, s);
        o += step;
    }
    for (int k = 0; k < left; k++) {
        *o = 0;
        o += step;
    }
}

// ---------------------------------------------------------------------------
// Spread
//
// One block per SM walks the items; an item is up to kTcK sources of one tile
// of (kTcX - P) x (kTcY - P) stencil origins, whose stencils lie in a patch of
// kTcX x kTcY nodes.  Two grids at a time (a "group") are rows 0..63 and
// 64..127 of the product: A = digits of c X (128 rows x sources, built 16
// sources at a time by one of two warpgroups), B = digits of Y (kept for the
// item, digit by digit along N), D = the levels, kTcY columns each, in TMEM.
// Digit p of A times B's digits 0 .. NS-1-p lands in levels p .. NS-1, so one
// instruction sequence per digit p of N = kTcY (NS - p) columns accumulates
// them all.  A ninth warp issues the products; the others build the next
// operands meanwhile, then combine the levels and add the patch to the grid.
// A tenth loads the next item's sources.
//
// Bound: latency between the phases of an item with two blocks per SM (issue 38 %,
// tensor pipe 21 % active).  2^20 sources, 2688^2 nodes, five grids: 1.70 ms (and
// 0.11 ms to sort the sources into tiles) against k_spread_fix's 4.67 ms, which is
// bound by its 3125 L2 atomics per source; here a source costs 222, in bulk
// reductions of one row of nodes each.  One block per SM with patches of 64 x 48
// nodes and items of 160 sources took 1.97 ms; 64-bit atomics from the threads in
// place of the bulk reductions 2.65 ms; bulk tensor reductions (64 rows in one
// instruction) the same as one per row.
// ---------------------------------------------------------------------------
constexpr int kTcBuild = 256, kTcThreads = kTcBuild + 64;
constexpr int kTcCols = 256;                         // TMEM columns

__host__ __device__ constexpr int tc_a_bytes(int NS) { return NS * 4096; }         // 16 sources
__host__ __device__ constexpr int tc_b_bytes(int NS) { return NS * kTcY * kTcK * 2; }
constexpr int kTcStageRow = kTcY * 8 + 16;           // the epilogue's staging: bytes per row of nodes
constexpr int kTcStage = 128 * kTcStageRow;
// A stencil's nodes lie in a window of whole 8-node chunks of its patch.
__host__ __device__ inline int tc_window(int P) { return (P + 7) / 8 * 8 + 8; }

// An item's sources as the loader warp leaves them (one item ahead).
struct TcSources {
    unsigned long long c[5][kTcK];                   // |c| / 2^ec as fractions of 2^63
    int meta[kTcK];
    unsigned char neg[5][kTcK];                      // the coefficients' signs
    int ec[5];
};

struct TcSmem {                                      // after the operand regions
    TcSources src[2];
    unsigned long long seed[6][kTcK];                // ex, ey, qpx, qpy, qmx, qmy
    unsigned long long full[2], free[2], done, tfree, fin, ready, sfree[2], seedfree;
    uint32_t tmem;
    int abort_flag;
};

static int tc_spread_smem(int NS, int P)
{
    const int w = tc_window(P) * kTcK * 8;
    const int a = std::max(std::max(2 * tc_a_bytes(NS), kTcStage), w);
    return a + tc_b_bytes(NS) + w + (int)sizeof(TcSmem) + 128;
}

template <int NC, int NS>
__global__ void __launch_bounds__(kTcThreads, 2) k_spread_tc(TcSpreadArgs a)
{
    chain_enter();
    static_assert(NS == kTcDigits && NS == 7, "the epilogue combines levels 0 .. 6");
    constexpr int NG = (NC + 1) / 2;
    constexpr int kBK = NS * (kTcY / 8) * 128;       // B: bytes per 8 sources
    extern __shared__ __align__(128) char tc_smem[];
    const unsigned long long bnd = *a.bound;
    if (bnd == kFixedOff) return;                    // the FP64 spread runs instead
    const int nit = *a.nitems;
    // few items: the groups of one item go to different blocks
    const bool split = nit < (int)gridDim.x;
    const int nv = split ? nit * NG : nit;
    // each block takes one run of the items: blocks at work at the same time are
    // then on distant tiles, whose patches do not overlap
    const int v0 = (int)((int64_t)nv * blockIdx.x / gridDim.x);
    const int v1 = (int)((int64_t)nv * (blockIdx.x + 1) / gridDim.x);
    if (v0 == v1) return;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int P = a.P, P1 = P + 1, win = tc_window(P), wbytes = win * kTcK * 8;
    const int abytes = max(max(2 * tc_a_bytes(NS), kTcStage), wbytes);
    char *Ash = tc_smem, *Bsh = Ash + abytes;
    unsigned long long *xs = reinterpret_cast<unsigned long long *>(Bsh + tc_b_bytes(NS));
    unsigned long long *ys = reinterpret_cast<unsigned long long *>(Ash);
    TcSmem &sh = *reinterpret_cast<TcSmem *>(reinterpret_cast<char *>(xs) + wbytes);
    volatile int *ab = &sh.abort_flag;

    if (tid == 0) {
        sh.abort_flag = 0;
        mbar_init(smem_u32(&sh.full[0]), kTcBuild / 2);
        mbar_init(smem_u32(&sh.full[1]), kTcBuild / 2);
        mbar_init(smem_u32(&sh.free[0]), 1);
        mbar_init(smem_u32(&sh.free[1]), 1);
        mbar_init(smem_u32(&sh.done), 1);
        mbar_init(smem_u32(&sh.tfree), kTcBuild);
        mbar_init(smem_u32(&sh.fin), 1);
        mbar_init(smem_u32(&sh.ready), 1);
        mbar_init(smem_u32(&sh.sfree[0]), kTcBuild);
        mbar_init(smem_u32(&sh.sfree[1]), kTcBuild);
        mbar_init(smem_u32(&sh.seedfree), kTcBuild);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kTcBuild / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sh.tmem)),
                     "n"(kTcCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    const int S = fix_shift(bnd);

    if (warp == kTcBuild / 32) {
        if (lane == 0) {
            int nfull[2] = {0, 0}, ng = 0;
            bool ok = true;
            for (int v = v0; v < v1 && ok; v++) {
                const int4 item = a.items[split ? v / NG : v];
                const int nk = (item.z + 15) >> 4;
                const int g0 = split ? v % NG : 0, g1 = split ? g0 + 1 : NG;
                for (int g = g0; g < g1 && ok; g++, ng++) {
                    for (int k = 0; k < nk; k++) {
                        const int b = k & 1;
                        ok = mbar_wait(smem_u32(&sh.full[b]), nfull[b]++ & 1, ab, a.wait) &&
                             !(k == 0 && ng > 0 && !mbar_wait(smem_u32(&sh.tfree), (ng - 1) & 1, ab, a.wait));
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t Aa = smem_u32(Ash) + b * tc_a_bytes(NS);
                        const uint32_t Ba = smem_u32(Bsh) + k * 2 * kBK;
#pragma unroll
                        for (int p = 0; p < NS; p++) {
                            const uint64_t da = tc_desc(Aa + p * 4096, 2048, 128);
                            tc_mma(tmem + kTcY * p, da, tc_desc(Ba, kBK, 128), tc_idesc(kTcY * (NS - p), 1),
                                   k > 0 || p > 0);
                        }
                        tc_commit(smem_u32(&sh.free[b]));
                    }
                    if (ok) tc_commit(smem_u32(&sh.done));
                }
            }
            tc_drain(smem_u32(&sh.fin), a.wait);
        }
        __syncwarp();
    } else if (warp == kTcBuild / 32 + 1) {
        // loader: the next item's offsets, seeds and coefficients, the
        // latter as integers at the power-of-two scale of the item's largest
        int n = 0;
        for (int v = v0; v < v1; v++, n++) {
            const int4 item = a.items[split ? v / NG : v];
            const int b = n & 1;
            TcSources &q = sh.src[b];
            const TcPoint *f[kTcK / 32];
            double cf[kTcK / 32][NC];
            int meta[kTcK / 32];
#pragma unroll
            for (int u = 0; u < kTcK / 32; u++) {
                const int s = lane + 32 * u;
                f[u] = nullptr;
                meta[u] = 0;
                if (s < item.z) {
                    const int j = a.list[item.y + s];
                    f[u] = reinterpret_cast<const TcPoint *>(a.fac) + j;
                    meta[u] = f[u]->meta;
#pragma unroll
                    for (int c = 0; c < NC; c++) cf[u][c] = a.coef[(int64_t)NC * j + c];
                } else {
#pragma unroll
                    for (int c = 0; c < NC; c++) cf[u][c] = 0.0;
                }
            }
            if (n > 1 && !__all_sync(~0u, mbar_wait(smem_u32(&sh.sfree[b]), (n / 2 - 1) & 1, ab, a.wait))) break;
#pragma unroll
            for (int u = 0; u < kTcK / 32; u++) q.meta[lane + 32 * u] = meta[u];
#pragma unroll
            for (int c = 0; c < NC; c++) {
                unsigned long long m = 0;
#pragma unroll
                for (int u = 0; u < kTcK / 32; u++)
                    m = max(m, (unsigned long long)__double_as_longlong(cf[u][c]) & 0x7fffffffffffffffull);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(~0u, m, o));
                const int ec = max((int)(m >> 52), 1) - 1022;     // |c| < 2^ec
                if (lane == 0) q.ec[c] = ec;
#pragma unroll
                for (int u = 0; u < kTcK / 32; u++) {
                    const unsigned long long w = (unsigned long long)__double_as_longlong(cf[u][c]);
                    const int e = (int)(w >> 52) & 0x7ff;
                    const unsigned long long t = (w & 0xfffffffffffffull) | (e ? 1ull << 52 : 0);
                    const int sh10 = max(e, 1) - 1012 - ec;      // |c| 2^(63 - ec) = t 2^sh10
                    q.c[c][lane + 32 * u] = sh10 >= 0 ? t << sh10 : sh10 > -54 ? (t + (1ull << (-sh10 - 1))) >> -sh10 : 0;
                    q.neg[c][lane + 32 * u] = (unsigned char)(w >> 63);
                }
            }
            if (n > 0 && !__all_sync(~0u, mbar_wait(smem_u32(&sh.seedfree), (n - 1) & 1, ab, a.wait))) break;
#pragma unroll
            for (int u = 0; u < kTcK / 32; u++) {
                if (!f[u]) continue;
                const int s = lane + 32 * u;
                sh.seed[0][s] = f[u]->ex;
                sh.seed[1][s] = f[u]->ey;
                sh.seed[2][s] = f[u]->qpx;
                sh.seed[3][s] = f[u]->qpy;
                sh.seed[4][s] = f[u]->qmx;
                sh.seed[5][s] = f[u]->qmy;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sh.ready));
        }
    } else {
        const int wg = tid / (kTcBuild / 2), wt = tid & (kTcBuild / 2 - 1);   // operand buffer, thread in it
        int nfill = 0, ng = 0, n = 0;
        const __half2 one = __float2half2_rn(1.0f), mone = __float2half2_rn(-1.0f);
        auto bstop = [&] { return tc_stop<1, kTcBuild>(ab); };
        bool stop = false;
        for (int v = v0; v < v1 && !stop; v++, n++) {
            const int4 item = a.items[split ? v / NG : v];
            const int g0 = split ? v % NG : 0, g1 = split ? g0 + 1 : NG;
            const int cnt = item.z, nk = (cnt + 15) >> 4, KP = nk * 16;
            const TcSources &src = sh.src[n & 1];
            const bool have = mbar_wait(smem_u32(&sh.ready), n & 1, ab, a.wait);
            // the factors along x and y, outward from the nearest node on both
            // sides, in the chunk-aligned windows of the stencils
            for (int t = have ? tid : 4 * kTcK; t < 4 * kTcK; t += kTcBuild) {
                const int q = t / kTcK, ax = q & 1, s = t % kTcK;
                if (s >= cnt) continue;
                const int meta = src.meta[s], ic = P / 2 + ((meta >> (16 + ax)) & 1);
                const int r = (meta >> (8 * ax)) & 7;
                const unsigned long long e = sh.seed[ax][s];
                unsigned long long *o = (ax ? ys : xs) + s;
                if (q < 2) {
                    tc_factors<kTcK>(e, sh.seed[2 + ax][s], a.s, r + ic, 1, P1 - ic, win, o);
                } else {
                    const unsigned long long qm = sh.seed[4 + ax][s];
                    tc_factors<kTcK>(mulhi_apx(e, qm), mulhi_apx(qm, a.s), a.s, r + ic - 1, -1, ic, win, o);
                }
            }
            mbar_arrive(smem_u32(&sh.seedfree));
            if (bstop()) break;
            // B: the digits of Y, four nodes of one source per step (the
            // window's chunks first, so that a warp's lanes agree)
            for (int t = tid; t < kTcK * (kTcY / 4); t += kTcBuild) {
                const int slot = t / (2 * kTcK), s = (t >> 1) % kTcK, half = t & 1;
                if (s >= KP) continue;
                int ch = ((src.meta[s] >> 11) & 31) + slot;
                if (ch >= kTcY / 8) ch -= kTcY / 8;
                char *dst = Bsh + (s >> 3) * kBK + ch * 128 + (s & 7) * 16 + half * 8;
                if (s >= cnt || 8 * slot >= win) {
                    store_zero_digits<NS>(dst, kTcY / 8 * 128);
                } else {
                    unsigned long long w[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) w[e] = ys[(8 * slot + 4 * half + e) * kTcK + s] >> 1;
                    store_digits<NS>(w, one, dst, kTcY / 8 * 128);
                }
            }
            fence_async_shared();
            if (bstop()) break;
            for (int g = g0; g < g1; g++, ng++) {
                bool ok = true;
                for (int k = wg; k < nk; k += 2) {
                    ok = nfill == 0 || mbar_wait(smem_u32(&sh.free[wg]), (nfill - 1) & 1, ab, a.wait);
                    if (!ok) break;
                    nfill++;
                    // A: 16 sources x two grids x 16 half chunks of 4 nodes,
                    // the window's in the loop's first pass
                    const int half = wt & 1, s = k * 16 + ((wt >> 1) & 15), gc = (wt >> 5) & 1, c = 2 * g + gc;
                    if (c < NC) {
                        const unsigned long long ci = src.c[c][s];
                        const __half2 sign = src.neg[c][s] ? mone : one;
                        const int ch0 = (src.meta[s] >> 3) & 31;
                        char *dst0 = Ash + wg * tc_a_bytes(NS) + ((s >> 3) & 1) * 2048 + gc * 1024 +
                                     (s & 7) * 16 + half * 8;
#pragma unroll 1
                        for (int slot = wt >> 6; slot < 8; slot += kTcBuild / 128) {
                            char *dst = dst0 + ((ch0 + slot) & 7) * 128;
                            if (8 * slot >= win || s >= cnt) {
                                store_zero_digits<NS>(dst, 4096);
                            } else {
                                unsigned long long w[4];
#pragma unroll
                                for (int e = 0; e < 4; e++)
                                    w[e] = mulhi_apx(ci, xs[(8 * slot + 4 * half + e) * kTcK + s]);
                                store_digits<NS>(w, sign, dst, 4096);
                            }
                        }
                    }
                    fence_async_shared();
                    mbar_arrive(smem_u32(&sh.full[wg]));
                }
                // the levels -> int64 at the grid's scale -> staging -> grid
                ok = __all_sync(~0u, ok && mbar_wait(smem_u32(&sh.done), ng & 1, ab, a.wait));
                tc_fence_after();
                const int quad = warp & 3, row = quad * 32 + lane, c = 2 * g + (quad >> 1);
                if (ok && c < NC) {
                    // c X Y 2^S = (H 2^32 + L) 2^-sh_n, sh_n > 0: H levels 0 .. 2, L levels 3 .. 6
                    const int sh_n = 62 - S - src.ec[c], sh_m = min(sh_n - 32, 60);
                    const long long round = 1ll << ((sh_n <= 32 ? sh_n : sh_m) - 1);
#pragma unroll 1
                    for (int yb = 0; yb < 2; yb++) {
                        const int y = (warp >> 2) * 16 + yb * 8;
                        uint32_t r[NS][8];
#pragma unroll
                        for (int l = 0; l < NS; l++)
                            tc_ld8(tmem + ((uint32_t)(quad * 32) << 16) + kTcY * l + y, r[l]);
#pragma unroll
                        for (int l = 0; l < NS; l++) tc_ld_wait8(r[l]);
#pragma unroll
                        for (int q = 0; q < 8; q += 2) {
                            long long o[2];
#pragma unroll
                            for (int e = 0; e < 2; e++) {
                                auto d = [&](int l) { return __float2int_rn(__uint_as_float(r[l][q + e])); };
                                const int p12 = d(1) * 256 + d(2), p34 = d(3) * 256 + d(4), p56 = d(5) * 256 + d(6);
                                const long long H = (long long)d(0) * 65536 + p12, L = (long long)p34 * 65536 + p56;
                                if (sh_n <= 32)
                                    o[e] = (H << (32 - sh_n)) + ((L + round) >> sh_n);
                                else
                                    o[e] = (H + (L >> 32) + round) >> sh_m;
                            }
                            *reinterpret_cast<longlong2 *>(Ash + row * kTcStageRow + (y + q) * 8) =
                                make_longlong2(o[0], o[1]);
                        }
                    }
                }
                tc_fence_before();
                mbar_arrive(smem_u32(&sh.tfree));
                if (g == g1 - 1) mbar_arrive(smem_u32(&sh.sfree[n & 1]));
                fence_async_shared();
                stop = bstop();
                if (stop) break;
                // one bulk reduction per row of nodes (two where it wraps)
                if (tid < 128 && 2 * g + (tid >> 6) < NC) {
                    int x = item.x / a.nty * a.Tx + (tid & 63);
                    if (x >= a.Mx) x -= a.Mx;
                    const int y = item.x % a.nty * a.Ty, m = min(kTcY, a.My - y);
                    long long *col = a.grid + ((int64_t)(2 * g + (tid >> 6)) * a.Mx + x) * a.My;
                    const uint32_t src = smem_u32(Ash) + tid * kTcStageRow;
                    bulk_add_u64(col + y, src, m * 8);
                    if (m < kTcY) bulk_add_u64(col, src + m * 8, (kTcY - m) * 8);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                }
                stop = bstop();
                if (stop) break;
            }
        }
        if (tid < 128) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kTcBuild / 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTcCols) : "memory");
}

// ---------------------------------------------------------------------------
// Gather
//
// u_c(t) = sum_i X_t[i] sum_j G_c[i][j] Y_t[j]: the inner sums of a tile's targets
// are a matrix product of Y (targets x nodes along y) with a patch of G_c.  An item
// is up to kTgT targets of one tile of (kTgX - P) x (kTgY - P) stencil origins, whose
// stencils lie in a patch of kTgX x kTgY nodes.  A = digits of Y (K-major, a row
// per target, kept for the item; rows 64 .. 127 of the product read what follows in
// shared memory and are ignored), B = digits of the patch of one grid, digit by
// digit along N, D = the levels, kTgX columns each.  The levels give the inner sums as
// int64, and each target's thread finishes with the X factors.  Warps whose TMEM
// lanes hold targets do that while the others build the next grid's B; a ninth
// issues the products, a tenth loads the next item's targets.
//
// Bound: tensor pipe (37 % active: 64 of the product's 128 rows hold targets, about
// 46 of them at 7 nodes per target) and the latency between an item's phases, two
// blocks per SM.  2^20 targets, 2688^2 nodes, four grids: 1.53 ms (and 0.09 ms
// to sort the targets into tiles) against k_gather_fix's 2.94 ms, bound by L1.
// ---------------------------------------------------------------------------
constexpr int kTgA = kTcDigits * kTgT * kTgY * 2, kTgB = kTcDigits * kTgX * kTgY * 2;
constexpr int kTgXs = kTgX * kTgT * 8;

struct TgSmem {
    unsigned long long seed[6][kTgT];
    int meta[2][kTgT], idx[2][kTgT];
    long long part[kTgT];
    unsigned long long bfull, done, tfree, fin, ready, sfree[2], seedfree;
    uint32_t tmem;
    int abort_flag;
};

constexpr int kTgSmem = kTgA + kTgB + kTgXs + (int)sizeof(TgSmem) + 128;

// Digits of eight signed numbers below 2^62 (all bytes biased), as store_digits.
__device__ __forceinline__ void store_digits_signed(const long long (&v)[8], char *dst, int stride)
{
    const __half2 off = __float2half2_rn(-1152.0f);
    uint32_t out[8][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const unsigned long long a = (unsigned long long)v[2 * k] + 0x8080808080808080ull;
        const unsigned long long b = (unsigned long long)v[2 * k + 1] + 0x8080808080808080ull;
#pragma unroll
        for (int w = 0; w < 2; w++) {
            const uint32_t aw = (uint32_t)(w ? a : a >> 32), bw = (uint32_t)(w ? b : b >> 32);
            const uint32_t z = __byte_perm(aw, bw, 0x7632), y = __byte_perm(aw, bw, 0x5410);
            const uint32_t d[4] = {__byte_perm(z, 0x64646464u, 0x4341), __byte_perm(z, 0x64646464u, 0x4240),
                                   __byte_perm(y, 0x64646464u, 0x4341), __byte_perm(y, 0x64646464u, 0x4240)};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const __half2 h = __hadd2(*reinterpret_cast<const __half2 *>(&d[q]), off);
                out[4 * w + q][k] = *reinterpret_cast<const uint32_t *>(&h);
            }
        }
    }
#pragma unroll
    for (int p = 0; p < kTcDigits; p++)
        *reinterpret_cast<uint4 *>(dst + p * stride) = make_uint4(out[p][0], out[p][1], out[p][2], out[p][3]);
}

// The same for four.
__device__ __forceinline__ void store_digits_signed4(const long long (&v)[4], char *dst, int stride)
{
    const __half2 off = __float2half2_rn(-1152.0f);
    uint32_t out[8][2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const unsigned long long a = (unsigned long long)v[2 * k] + 0x8080808080808080ull;
        const unsigned long long b = (unsigned long long)v[2 * k + 1] + 0x8080808080808080ull;
#pragma unroll
        for (int w = 0; w < 2; w++) {
            const uint32_t aw = (uint32_t)(w ? a : a >> 32), bw = (uint32_t)(w ? b : b >> 32);
            const uint32_t z = __byte_perm(aw, bw, 0x7632), y = __byte_perm(aw, bw, 0x5410);
            const uint32_t d[4] = {__byte_perm(z, 0x64646464u, 0x4341), __byte_perm(z, 0x64646464u, 0x4240),
                                   __byte_perm(y, 0x64646464u, 0x4341), __byte_perm(y, 0x64646464u, 0x4240)};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const __half2 h = __hadd2(*reinterpret_cast<const __half2 *>(&d[q]), off);
                out[4 * w + q][k] = *reinterpret_cast<const uint32_t *>(&h);
            }
        }
    }
#pragma unroll
    for (int p = 0; p < kTcDigits; p++)
        *reinterpret_cast<uint2 *>(dst + p * stride) = make_uint2(out[p][0], out[p][1]);
}

template <int NC>
__global__ void __launch_bounds__(kTcThreads, 2) k_gather_tc(TcGatherArgs a)
{
    chain_enter();
    extern __shared__ __align__(128) char tc_smem[];
    if (gmax_all(a.gmax) >= kGridNonFinite) return;  // the FP64 gather runs instead
    const int nv = *a.nitems;
    const int v0 = (int)((int64_t)nv * blockIdx.x / gridDim.x);
    const int v1 = (int)((int64_t)nv * (blockIdx.x + 1) / gridDim.x);
    if (v0 == v1) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int P = a.P, P1 = P + 1, win = tc_window(P);
    char *Ash = tc_smem, *Bsh = Ash + kTgA;
    unsigned long long *xs = reinterpret_cast<unsigned long long *>(Bsh + kTgB);
    unsigned long long *ys = reinterpret_cast<unsigned long long *>(Bsh);
    TgSmem &sh = *reinterpret_cast<TgSmem *>(reinterpret_cast<char *>(xs) + kTgXs);
    volatile int *ab = &sh.abort_flag;

    if (tid == 0) {
        sh.abort_flag = 0;
        mbar_init(smem_u32(&sh.bfull), 128);
        mbar_init(smem_u32(&sh.done), 1);
        mbar_init(smem_u32(&sh.tfree), 128);
        mbar_init(smem_u32(&sh.fin), 1);
        mbar_init(smem_u32(&sh.ready), 1);
        mbar_init(smem_u32(&sh.sfree[0]), kTcBuild);
        mbar_init(smem_u32(&sh.sfree[1]), kTcBuild);
        mbar_init(smem_u32(&sh.seedfree), kTcBuild);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kTcBuild / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sh.tmem)),
                     "n"(kTcCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;

    if (warp == kTcBuild / 32) {
        if (lane == 0) {
            int n = 0;
            bool ok = true;
            for (int v = v0; v < v1 && ok; v++) {
                for (int c = 0; c < NC; c++, n++) {
                    ok = mbar_wait(smem_u32(&sh.bfull), n & 1, ab, a.wait) &&
                         (n == 0 || mbar_wait(smem_u32(&sh.tfree), (n - 1) & 1, ab, a.wait));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int k = 0; k < kTgY / 16; k++)
#pragma unroll
                        for (int p = 0; p < kTcDigits; p++)
                            tc_mma(tmem + kTgX * p,
                                   tc_desc(smem_u32(Ash) + p * (kTgT * kTgY * 2) + k * 256, 128, kTgY * 16),
                                   tc_desc(smem_u32(Bsh) + k * 256, 128, kTgY * 16),
                                   tc_idesc(kTgX * (kTcDigits - p), 0), k > 0 || p > 0);
                    tc_commit(smem_u32(&sh.done));
                }
            }
            tc_drain(smem_u32(&sh.fin), a.wait);
        }
        __syncwarp();
    } else if (warp == kTcBuild / 32 + 1) {
        int n = 0;
        for (int v = v0; v < v1; v++, n++) {
            const int4 item = a.items[v];
            const int b = n & 1;
            const TcPoint *f[kTgT / 32];
            int meta[kTgT / 32], idx[kTgT / 32];
#pragma unroll
            for (int u = 0; u < kTgT / 32; u++) {
                const int s = lane + 32 * u;
                f[u] = nullptr;
                meta[u] = 0;
                idx[u] = -1;
                if (s < item.z) {
                    idx[u] = a.list[item.y + s];
                    f[u] = reinterpret_cast<const TcPoint *>(a.fac) + idx[u];
                    meta[u] = f[u]->meta;
                }
            }
            if (n > 1 && !__all_sync(~0u, mbar_wait(smem_u32(&sh.sfree[b]), (n / 2 - 1) & 1, ab, a.wait))) break;
#pragma unroll
            for (int u = 0; u < kTgT / 32; u++) {
                sh.meta[b][lane + 32 * u] = meta[u];
                sh.idx[b][lane + 32 * u] = idx[u];
            }
            if (n > 0 && !__all_sync(~0u, mbar_wait(smem_u32(&sh.seedfree), (n - 1) & 1, ab, a.wait))) break;
#pragma unroll
            for (int u = 0; u < kTgT / 32; u++) {
                if (!f[u]) continue;
                const int s = lane + 32 * u;
                sh.seed[0][s] = f[u]->ex;
                sh.seed[1][s] = f[u]->ey;
                sh.seed[2][s] = f[u]->qpx;
                sh.seed[3][s] = f[u]->qpy;
                sh.seed[4][s] = f[u]->qmx;
                sh.seed[5][s] = f[u]->qmy;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sh.ready));
        }
    } else {
        int n = 0, nc = 0;                           // items, grids so far
        const __half2 one = __float2half2_rn(1.0f);
        const bool epi = (warp & 2) == 0;            // TMEM lanes 0 .. 63: targets
        const int et = (warp & 1) * 32 + lane, eh = warp >> 2;            // target, half of the columns
        const int bt = ((warp >> 2) * 2 + (warp & 1)) * 32 + lane;        // builder thread
        auto bstop = [&] { return tc_stop<1, kTcBuild>(ab); };
        for (int v = v0; v < v1; v++, n++) {
            const int4 item = a.items[v];
            const int cnt = item.z, b = n & 1;
            const bool have = mbar_wait(smem_u32(&sh.ready), n & 1, ab, a.wait);
            // the factors: x in the patch's coordinates (as fractions of 2^62), y in
            // the chunk-aligned window (B's region holds them until A is built)
            for (int t = have ? tid : 4 * kTgT; t < 4 * kTgT; t += kTcBuild) {
                const int q = t / kTgT, ax = q & 1, s = t % kTgT;
                if (s >= cnt) continue;
                const int meta = sh.meta[b][s], ic = P / 2 + ((meta >> (16 + ax)) & 1);
                const int r = ax ? (meta >> 8) & 7 : meta & 0xff, w = ax ? win : kTgX;
                const unsigned long long e = ax ? sh.seed[1][s] : sh.seed[0][s] >> 2;
                unsigned long long *o = (ax ? ys : xs) + s;
                if (q < 2) {
                    tc_factors<kTgT>(e, sh.seed[2 + ax][s], a.s, r + ic, 1, P1 - ic, w, o);
                } else {
                    const unsigned long long qm = sh.seed[4 + ax][s];
                    tc_factors<kTgT>(mulhi_apx(e, qm), mulhi_apx(qm, a.s), a.s, r + ic - 1, -1, ic, w, o);
                }
            }
            mbar_arrive(smem_u32(&sh.seedfree));
            if (bstop()) break;
            for (int t = tid; t < kTgT * (kTgY / 4); t += kTcBuild) {
                const int slot = t / (2 * kTgT), s = (t >> 1) % kTgT, half = t & 1;
                const int ch = (((sh.meta[b][s] >> 11) & 31) + slot) & (kTgY / 8 - 1);
                char *dst = Ash + (s >> 3) * (kTgY * 16) + ch * 128 + (s & 7) * 16 + half * 8;
                if (s >= cnt || 8 * slot >= win) {
                    store_zero_digits<kTcDigits>(dst, kTgT * kTgY * 2);
                } else {
                    unsigned long long w[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) w[e] = ys[(8 * slot + 4 * half + e) * kTgT + s] >> 1;
                    store_digits<kTcDigits>(w, one, dst, kTgT * kTgY * 2);
                }
            }
            fence_async_shared();
            if (bstop()) break;
            const int x0 = item.x / a.nty * a.Tx, y0 = item.x % a.nty * a.Ty;
            long long first = 0;                     // the first of a pair's two sums
            for (int c = 0; c < NC; c++, nc++) {
                if (!epi) {
                    // B: 32 columns x 8 chunks of 8 nodes
                    if (c > 0 && !mbar_wait(smem_u32(&sh.done), (nc - 1) & 1, ab, a.wait)) break;
                    const long long *grid = a.grid + (int64_t)c * a.Mx * a.My;
#pragma unroll 1
                    for (int t = bt; t < kTgX * (kTgY / 8); t += 128) {
                        const int i = t % kTgX, ch = t / kTgX;
                        int x = x0 + i, y = y0 + 8 * ch;
                        if (x >= a.Mx) x -= a.Mx;
                        if (y >= a.My) y -= a.My;
                        const long long *g = grid + (int64_t)x * a.My;
                        long long w[8];
                        if (y + 8 <= a.My) {
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                const longlong2 q = __ldg(reinterpret_cast<const longlong2 *>(g + y) + e);
                                w[2 * e] = q.x;
                                w[2 * e + 1] = q.y;
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; e++) w[e] = __ldg(g + (y + e >= a.My ? y + e - a.My : y + e));
                        }
                        store_digits_signed(w, Bsh + (i >> 3) * (kTgY * 16) + ch * 128 + (i & 7) * 16, kTgX * kTgY * 2);
                    }
                    fence_async_shared();
                    mbar_arrive(smem_u32(&sh.bfull));
                } else {
                    const bool ok = __all_sync(~0u, mbar_wait(smem_u32(&sh.done), nc & 1, ab, a.wait));
                    tc_fence_after();
                    long long acc = 0;
#pragma unroll 1
                    for (int h = ok ? 0 : kTgX / 16; h < kTgX / 16; h++) {
                        const int i0 = eh * (kTgX / 2) + 8 * h;
                        uint32_t r[kTcDigits][8];
#pragma unroll
                        for (int l = 0; l < kTcDigits; l++)
                            tc_ld8(tmem + ((uint32_t)((warp & 1) * 32) << 16) + kTgX * l + i0, r[l]);
#pragma unroll
                        for (int l = 0; l < kTcDigits; l++) tc_ld_wait8(r[l]);
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            auto d = [&](int l) { return __float2int_rn(__uint_as_float(r[l][e])); };
                            const int p12 = d(1) * 256 + d(2), p34 = d(3) * 256 + d(4), p56 = d(5) * 256 + d(6);
                            const unsigned hi = (unsigned)d(0) * 65536u + (unsigned)p12;
                            const long long V = (long long)p34 * 65536 + p56 + (long long)((unsigned long long)hi << 32);
                            const unsigned long long x = xs[(i0 + e) * kTgT + et];
                            acc += (long long)mulhi_apx((unsigned long long)V, x) - (V < 0 ? (long long)x : 0);
                        }
                    }
                    tc_fence_before();
                    mbar_arrive(smem_u32(&sh.tfree));
                    // the two halves of the columns
                    if (eh) sh.part[et] = acc;
                    if (tc_stop<2, 128>(ab)) break;
                    if (!eh) {
                        acc += sh.part[et];
                        if (c & 1) {
                            const int j = sh.idx[b][et];
                            const unsigned long long gb = a.gmax[c / 2];
                            const double s = gb == 0 ? 0.0 : ldexp(a.scale, 3 - grid_shift(gb, a.Bg));
                            if (j >= 0)
                                a.out[(int64_t)(c / 2) * a.nt + j] = make_double2((double)first * s, (double)acc * s);
                        } else {
                            first = acc;
                        }
                    }
                    asm volatile("bar.sync 2, 128;" ::: "memory");
                }
            }
            mbar_arrive(smem_u32(&sh.sfree[b]));
            // the item's last product has read A and B (the epilogue waited for it)
            if (bstop()) break;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kTcBuild / 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTcCols) : "memory");
}

// ---------------------------------------------------------------------------
// Adjoint gather
//
// At each forward source, for the five adjoint grids: the value sum_ij X_i Y_j g and the
// sums with the weights' position derivatives, X'_i = 2 a h (u_x - i') X_i with i' the
// node's offset from the stencil's middle and u_x the point's in nodes, and the
// same in y.  Rows 0 .. 63 of the product are Y, rows 64 .. 127 are j' Y for the same
// points, so one product gives sum_j Y_j g and sum_j j' Y_j g; the threads of the
// first rows also add i' X_i times their sums.  One block per SM, the accumulators
// and B doubled: while one grid is multiplied, the previous one's sums are
// finished and the next one's B is built.
//
// Bound: latency (one block of 18 warps per SM).  2^18 sources, 1344^2 nodes: 0.74 ms
// (and 0.09 ms for the tiles and the int64 grids) against 2.17 ms for
// k_gather_adj_ff with its float-float grids, bound by issue; 1500 sources on 96^2
// nodes 0.027 against 0.375 ms.  The gradients' error falls from 6e-14 to 4e-15
// with it, the weights no longer being float-float.
// ---------------------------------------------------------------------------
constexpr int kGaThreads = 18 * 32;
constexpr int kGaA = kTcDigits * 128 * kTgY * 2;

struct GaSmem {
    unsigned long long seed[6][kTgT];
    double coef[2][5][kTgT], ux[2][kTgT], uy[2][kTgT];
    int meta[2][kTgT], idx[2][kTgT];
    long long sum[2][5][128], sumx[2][5][kTgT];      // per half of the columns
    unsigned long long bfull[2], done[2], tfree[2], fin, ready, sfree[2], seedfree;
    uint32_t tmem;
    int abort_flag;
};

constexpr int kGaSmem = kGaA + 2 * kTgB + kTgXs + (int)sizeof(GaSmem) + 128;

__global__ void __launch_bounds__(kGaThreads, 1) k_gather_adj_tc(TcGatherAdjArgs a)
{
    chain_enter();
    extern __shared__ __align__(128) char tc_smem[];
    if (gmax_all(a.gmax) >= kGridNonFinite) return;  // the FP64 gather runs instead
    const int nv = *a.nitems;
    const int v0 = (int)((int64_t)nv * blockIdx.x / gridDim.x);
    const int v1 = (int)((int64_t)nv * (blockIdx.x + 1) / gridDim.x);
    if (v0 == v1) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int P = a.P, P1 = P + 1, win = tc_window(P);
    char *Ash = tc_smem, *Bsh = Ash + kGaA;
    unsigned long long *xs = reinterpret_cast<unsigned long long *>(Bsh + 2 * kTgB);
    unsigned long long *ys = reinterpret_cast<unsigned long long *>(Bsh);
    GaSmem &sh = *reinterpret_cast<GaSmem *>(reinterpret_cast<char *>(xs) + kTgXs);
    volatile int *ab = &sh.abort_flag;

    if (tid == 0) {
        sh.abort_flag = 0;
        for (int b = 0; b < 2; b++) {
            mbar_init(smem_u32(&sh.bfull[b]), 256);
            mbar_init(smem_u32(&sh.done[b]), 1);
            mbar_init(smem_u32(&sh.tfree[b]), 256);
            mbar_init(smem_u32(&sh.sfree[b]), 512);
        }
        mbar_init(smem_u32(&sh.fin), 1);
        mbar_init(smem_u32(&sh.ready), 1);
        mbar_init(smem_u32(&sh.seedfree), 256);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&sh.tmem))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;

    if (warp == 16) {
        if (lane == 0) {
            int n = 0;
            bool ok = true;
            for (int v = v0; v < v1 && ok; v++) {
                for (int c = 0; c < 5; c++, n++) {
                    const int b = n & 1;
                    ok = mbar_wait(smem_u32(&sh.bfull[b]), (n >> 1) & 1, ab, a.wait) &&
                         (n <= 1 || mbar_wait(smem_u32(&sh.tfree[b]), ((n >> 1) - 1) & 1, ab, a.wait));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int k = 0; k < kTgY / 16; k++)
#pragma unroll
                        for (int p = 0; p < kTcDigits; p++)
                            tc_mma(tmem + 256 * b + kTgX * p,
                                   tc_desc(smem_u32(Ash) + p * (128 * kTgY * 2) + k * 256, 128, kTgY * 16),
                                   tc_desc(smem_u32(Bsh) + b * kTgB + k * 256, 128, kTgY * 16),
                                   tc_idesc(kTgX * (kTcDigits - p), 0), k > 0 || p > 0);
                    tc_commit(smem_u32(&sh.done[b]));
                }
            }
            tc_drain(smem_u32(&sh.fin), a.wait);
        }
        __syncwarp();
    } else if (warp == 17) {
        int n = 0;
        for (int v = v0; v < v1; v++, n++) {
            const int4 item = a.items[v];
            const int b = n & 1;
            if (n > 1 && !__all_sync(~0u, mbar_wait(smem_u32(&sh.sfree[b]), (n / 2 - 1) & 1, ab, a.wait))) break;
            const TcPoint *f[kTgT / 32];
#pragma unroll
            for (int u = 0; u < kTgT / 32; u++) {
                const int s = lane + 32 * u;
                f[u] = nullptr;
                int j = -1, meta = 0;
                if (s < item.z) {
                    j = a.list[item.y + s];
                    f[u] = reinterpret_cast<const TcPoint *>(a.fac) + j;
                    meta = f[u]->meta;
#pragma unroll
                    for (int c = 0; c < 5; c++) sh.coef[b][c][s] = a.coef[5 * (int64_t)j + c];
                    const double2 S = a.sp[j];
                    int mx, my;
                    double px, py;
                    closest_node(S.x, S.y, a.Lhx, a.Lhy, a.h, P, mx, my, px, py);
                    sh.ux[b][s] = px / a.h;
                    sh.uy[b][s] = py / a.h;
                }
                sh.meta[b][s] = meta;
                sh.idx[b][s] = j;
            }
            if (n > 0 && !__all_sync(~0u, mbar_wait(smem_u32(&sh.seedfree), (n - 1) & 1, ab, a.wait))) break;
#pragma unroll
            for (int u = 0; u < kTgT / 32; u++) {
                if (!f[u]) continue;
                const int s = lane + 32 * u;
                sh.seed[0][s] = f[u]->ex;
                sh.seed[1][s] = f[u]->ey;
                sh.seed[2][s] = f[u]->qpx;
                sh.seed[3][s] = f[u]->qpy;
                sh.seed[4][s] = f[u]->qmx;
                sh.seed[5][s] = f[u]->qmy;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sh.ready));
        }
    } else {
        int n = 0, nc = 0;                           // items, grids so far
        const __half2 one = __float2half2_rn(1.0f);
        auto bstop = [&] { return tc_stop<1, 512>(ab); };
        for (int v = v0; v < v1; v++, n++) {
            const int4 item = a.items[v];
            const int cnt = item.z, b = n & 1;
            const bool have = mbar_wait(smem_u32(&sh.ready), n & 1, ab, a.wait);
            if (tid < 4 * kTgT) {
                const int q = tid / kTgT, ax = q & 1, s = tid % kTgT;
                if (have && s < cnt) {
                    const int meta = sh.meta[b][s], ic = P / 2 + ((meta >> (16 + ax)) & 1);
                    const int r = ax ? (meta >> 8) & 7 : meta & 0xff, w = ax ? win : kTgX;
                    const unsigned long long e = ax ? sh.seed[1][s] : sh.seed[0][s] >> 2;
                    unsigned long long *o = (ax ? ys : xs) + s;
                    if (q < 2) {
                        tc_factors<kTgT>(e, sh.seed[2 + ax][s], a.s, r + ic, 1, P1 - ic, w, o);
                    } else {
                        const unsigned long long qm = sh.seed[4 + ax][s];
                        tc_factors<kTgT>(mulhi_apx(e, qm), mulhi_apx(qm, a.s), a.s, r + ic - 1, -1, ic, w, o);
                    }
                }
                mbar_arrive(smem_u32(&sh.seedfree));
            }
            if (bstop()) break;
            for (int t = tid; t < 2 * kTgT * (kTgY / 4); t += 512) {
                const int der = t / (kTgT * (kTgY / 4)), t1 = t % (kTgT * (kTgY / 4));
                const int slot = t1 / (2 * kTgT), s = (t1 >> 1) % kTgT, half = t1 & 1, row = 64 * der + s;
                const int oy = (sh.meta[b][s] >> 8) & 0xff;
                const int ch = ((oy >> 3) + slot) & (kTgY / 8 - 1);
                char *dst = Ash + (row >> 3) * (kTgY * 16) + ch * 128 + (row & 7) * 16 + half * 8;
                if (s >= cnt || 8 * slot >= win) {
                    store_zero_digits<kTcDigits>(dst, 128 * kTgY * 2);
                } else {
                    unsigned long long w[4];
                    const int r0 = 8 * slot + 4 * half;
#pragma unroll
                    for (int e = 0; e < 4; e++) w[e] = ys[(r0 + e) * kTgT + s] >> 1;
                    if (der) {
                        // j' Y as fractions of 2^61 (|j' Y| < 2)
                        const int j0 = r0 - (oy & 7) - P / 2;
                        long long z[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) z[e] = (long long)(w[e] >> 2) * (j0 + e);
                        store_digits_signed4(z, dst, 128 * kTgY * 2);
                    } else {
                        store_digits<kTcDigits>(w, one, dst, 128 * kTgY * 2);
                    }
                }
            }
            fence_async_shared();
            if (bstop()) break;
            const int x0 = item.x / a.nty * a.Tx, y0 = item.x % a.nty * a.Ty;
            for (int c = 0; c < 5; c++, nc++) {
                const int tb = nc & 1;
                if (warp >= 8) {
                    // B: 32 columns x 8 chunks of 8 nodes, one each
                    if (nc > 1 && !mbar_wait(smem_u32(&sh.done[tb]), ((nc >> 1) - 1) & 1, ab, a.wait)) break;
                    const int bt = tid - 256, i = bt % kTgX, ch = bt / kTgX;
                    int x = x0 + i, y = y0 + 8 * ch;
                    if (x >= a.Mx) x -= a.Mx;
                    if (y >= a.My) y -= a.My;
                    const long long *g = a.grid + ((int64_t)c * a.Mx + x) * a.My;
                    long long w[8];
                    if (y + 8 <= a.My) {
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const longlong2 q = __ldg(reinterpret_cast<const longlong2 *>(g + y) + e);
                            w[2 * e] = q.x;
                            w[2 * e + 1] = q.y;
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; e++) w[e] = __ldg(g + (y + e >= a.My ? y + e - a.My : y + e));
                    }
                    store_digits_signed(w, Bsh + tb * kTgB + (i >> 3) * (kTgY * 16) + ch * 128 + (i & 7) * 16,
                                        kTgX * kTgY * 2);
                    fence_async_shared();
                    mbar_arrive(smem_u32(&sh.bfull[tb]));
                } else {
                    const int quad = warp & 3, eh = warp >> 2, t = (quad & 1) * 32 + lane;
                    const int mid = (sh.meta[b][t] & 0xff) + P / 2;
                    if (!__all_sync(~0u, mbar_wait(smem_u32(&sh.done[tb]), (nc >> 1) & 1, ab, a.wait))) break;
                    tc_fence_after();
                    long long acc = 0, accx = 0;
#pragma unroll 1
                    for (int h = 0; h < kTgX / 16; h++) {
                        const int i0 = eh * (kTgX / 2) + 8 * h;
                        uint32_t r[kTcDigits][8];
#pragma unroll
                        for (int l = 0; l < kTcDigits; l++)
                            tc_ld8(tmem + 256 * tb + ((uint32_t)(quad * 32) << 16) + kTgX * l + i0, r[l]);
#pragma unroll
                        for (int l = 0; l < kTcDigits; l++) tc_ld_wait8(r[l]);
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            auto d = [&](int l) { return __float2int_rn(__uint_as_float(r[l][e])); };
                            const int p12 = d(1) * 256 + d(2), p34 = d(3) * 256 + d(4), p56 = d(5) * 256 + d(6);
                            const unsigned hi = (unsigned)d(0) * 65536u + (unsigned)p12;
                            const long long V = (long long)p34 * 65536 + p56 + (long long)((unsigned long long)hi << 32);
                            const unsigned long long x = xs[(i0 + e) * kTgT + t];
                            const long long m = (long long)mulhi_apx((unsigned long long)V, x) - (V < 0 ? (long long)x : 0);
                            acc += m;
                            accx += (m >> 3) * (i0 + e - mid);
                        }
                    }
                    tc_fence_before();
                    mbar_arrive(smem_u32(&sh.tfree[tb]));
                    sh.sum[eh][c][quad * 32 + lane] = acc;
                    if (quad < 2) sh.sumx[eh][c][t] = accx;
                }
            }
            // (the item's last products have read A: the epilogue waited for them)
            if (bstop()) break;
            if (tid < cnt) {
                const int j = sh.idx[b][tid];
                const double ux = sh.ux[b][tid], uy = sh.uy[b][tid];
                double gx = 0.0, gy = 0.0;
                double *o = a.out + 7 * (int64_t)j;
#pragma unroll
                for (int c = 0; c < 5; c++) {
                    const unsigned long long gb = a.gmax[c / 2];
                    const double s = gb == 0 ? 0.0 : ldexp(a.scale, 3 - grid_shift(gb, a.Bg));
                    const double V = (double)(sh.sum[0][c][tid] + sh.sum[1][c][tid]) * s;
                    const double Ix = (double)(sh.sumx[0][c][tid] + sh.sumx[1][c][tid]) * (8.0 * s);
                    const double Iy = (double)(sh.sum[0][c][64 + tid] + sh.sum[1][c][64 + tid]) * (4.0 * s);
                    const double cf = sh.coef[b][c][tid];
                    o[c] = V;
                    gx = fma(cf, fma(ux, V, -Ix), gx);
                    gy = fma(cf, fma(uy, V, -Iy), gy);
                }
                o[5] = gx * a.dscale;
                o[6] = gy * a.dscale;
            }
            mbar_arrive(smem_u32(&sh.sfree[b]));
            if (bstop()) break;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 16)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
cudaError_t launch_tc_points(const TcPrepArgs &b, int nset, const unsigned long long *bound,
                             int nbound, int bstride, cudaStream_t st, int64_t &launches)
{
    int64_t n = 0;
    int ntile = 0;
    for (int k = 0; k < nset; k++) {
        n = b.s[k].a.n > n ? b.s[k].a.n : n;
        ntile = b.s[k].ntile > ntile ? b.s[k].ntile : ntile;
    }
    const dim3 g((unsigned)((n + 255) / 256), nset);
    if (n > 0) launch_chained(k_tc_points, g, 256, 0, st, b);
    launch_chained(k_tc_items, dim3((ntile + 1023) / 1024, nset), 1024, 0, st, b);
    if (n > 0) launch_chained(k_tc_list, g, 256, 0, st, b);
    launches += n > 0 ? 3 : 1;
    for (int k = 0; k < nset; k++) {
        const TcSetArgs &t = b.s[k];
        if (t.perm && t.a.n > 0) {
            const bool lg = t.a.n > kOrderFrom;
            launch_chained(k_tc_order, (unsigned)((t.a.n + 255) / 256), 256, 0, st, t.a.n, t.a.tile, t.start, t.kmax,
                           lg ? kOrderLong : INT_MAX, t.key, t.list, t.ordered, bound, nbound, bstride);
            launches++;
            if (lg) {
                launch_chained(k_tc_order_long, std::min(t.ntile, 2 * sm_count()), kOrderThreads, 0, st, t.a.n, t.ntile,
                               t.start, t.key, t.list, t.ordered, t.tmp, bound, nbound, bstride);
                launches++;
            }
        }
    }
    return cudaGetLastError();
}

template <int NC, int NS>
static cudaError_t spread_tc(const TcSpreadArgs &a, cudaStream_t st)
{
    // (the limit is the process's, not the launch's: that of the widest stencil, so that
    // another thread's call cannot lower it in between)
    const cudaError_t e = cudaFuncSetAttribute(k_spread_tc<NC, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               tc_spread_smem(NS, kTcMaxP));
    if (e != cudaSuccess) return e;
    launch_chained(k_spread_tc<NC, NS>, 2 * sm_count(), kTcThreads, tc_spread_smem(NS, a.P), st, a);
    return cudaGetLastError();
}

cudaError_t launch_spread_tc(const TcSpreadArgs &a, int nc, cudaStream_t st, int64_t &launches)
{
    launches++;
    switch (nc) {
    case 2: return spread_tc<2, kTcDigits>(a, st);
    case 3: return spread_tc<3, kTcDigits>(a, st);
    case 4: return spread_tc<4, kTcDigits>(a, st);
    default: return spread_tc<5, kTcDigits>(a, st);
    }
}

template <int NC>
static cudaError_t gather_tc(const TcGatherArgs &a, cudaStream_t st)
{
    const cudaError_t e =
        cudaFuncSetAttribute(k_gather_tc<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTgSmem);
    if (e != cudaSuccess) return e;
    launch_chained(k_gather_tc<NC>, 2 * sm_count(), kTcThreads, kTgSmem, st, a);
    return cudaGetLastError();
}

cudaError_t launch_gather_tc(const TcGatherArgs &a, int nc, cudaStream_t st, int64_t &launches)
{
    launches++;
    return nc == 2 ? gather_tc<2>(a, st) : gather_tc<4>(a, st);
}

cudaError_t launch_gather_adj_tc(const TcGatherAdjArgs &a, cudaStream_t st, int64_t &launches)
{
    const cudaError_t e =
        cudaFuncSetAttribute(k_gather_adj_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kGaSmem);
    if (e != cudaSuccess) return e;
    launch_chained(k_gather_adj_tc, sm_count(), kGaThreads, kGaSmem, st, a);
    launches++;
    return cudaGetLastError();
}

}  // namespace se2p
