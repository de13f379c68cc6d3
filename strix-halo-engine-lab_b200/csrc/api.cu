// The C ABI (include/b200moe.h): host-side validation and composition. Argument errors are reported before anything
// is enqueued; nothing here allocates, synchronises (except b200moe_ffn_host, which says so) or starts threads.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>

#include "kernels.cuh"

namespace b200moe {

std::string& last_error_slot() {
    thread_local std::string text;
    return text;
}
int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    last_error_slot() = buf;
    return code;
}
std::atomic<u64>& launch_counter() {
    static std::atomic<u64> n{0};
    return n;
}
const char*& last_launch_slot() {
    thread_local const char* name = "";
    return name;
}
int after_launch(const char* what) {
    last_launch_slot() = what;
    launch_counter().fetch_add(1, std::memory_order_relaxed);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(B200MOE_ERR_CUDA, "launch of %s failed: %s", what, cudaGetErrorString(e));
    return B200MOE_OK;
}
bool device_ready() {
    static std::once_flag once;
    static bool ok = false;
    static std::string why;
    std::call_once(once, [] {
        int n = 0;
        cudaError_t e = cudaGetDeviceCount(&n);
        if (e != cudaSuccess || n == 0) { why = std::string("no CUDA device: ") + cudaGetErrorString(e); cudaGetLastError(); return; }
        int dev = 0;
        cudaDeviceProp p{};
        if (cudaGetDevice(&dev) != cudaSuccess || cudaGetDeviceProperties(&p, dev) != cudaSuccess) { why = "cannot query the CUDA device"; return; }
        if (p.major != 10) { why = "this library holds sm_100a code only; device is sm_" + std::to_string(p.major * 10 + p.minor); return; }
        ok = true;
    });
    if (!ok) fail(B200MOE_ERR_CUDA, "%s (there is no CPU fallback)", why.c_str());
    return ok;
}

int device_sm_count() {  // asked of the runtime once a device
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices];
    int dev = 0, n = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return n;
    if (dev < kDevices && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
    n = 148;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && dev < kDevices) known[dev].store(n, std::memory_order_relaxed);
    return n;
}

int ensure_dynamic_smem(const void* kernel, u32 bytes) {
    // The 48 KiB a launch gets without opting in cover static AND dynamic shared memory, so a kernel's own static arrays decide
    // from which size on it has to opt in.
    static std::mutex m;
    static std::map<std::pair<int, const void*>, u32> granted;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(m);
    auto it = granted.find({dev, kernel});
    if (it == granted.end()) {
        cudaFuncAttributes a{};
        const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
        if (e != cudaSuccess) return fail(B200MOE_ERR_CUDA, "cudaFuncGetAttributes: %s", cudaGetErrorString(e));
        const u32 fixed = static_cast<u32>(a.sharedSizeBytes), plain = 48u * 1024u;
        it = granted.emplace(std::make_pair(dev, kernel), fixed < plain ? plain - fixed : 0u).first;
    }
    u32& have = it->second;
    if (bytes <= have) return B200MOE_OK;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e != cudaSuccess) return fail(B200MOE_ERR_CUDA, "cudaFuncSetAttribute(dynamic smem %u): %s", bytes, cudaGetErrorString(e));
    have = bytes;
    return B200MOE_OK;
}

// The decode step alternates kernels that need almost all of an SM's shared memory with kernels that need little. Asking
// for the largest shared-memory carve-out on the small ones too keeps the SMs' L1 / shared split the same from one
// kernel of the step to the next (a change of the split has to wait for the SM to drain). Once per kernel and device.
int prefer_max_shared(const void* kernel) {
    static std::mutex m;
    static std::map<std::pair<int, const void*>, bool> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(m);
    bool& set = done[{dev, kernel}];
    if (set) return B200MOE_OK;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, static_cast<int>(cudaSharedmemCarveoutMaxShared));
    if (e != cudaSuccess) return fail(B200MOE_ERR_CUDA, "cudaFuncSetAttribute(carve-out): %s", cudaGetErrorString(e));
    set = true;
    return B200MOE_OK;
}

namespace {
std::atomic<u32> g_debug[3] = {{0}, {0}, {0}};
}
u32 debug_value(u32 key) { return key < 3 ? g_debug[key].load(std::memory_order_relaxed) : 0u; }

u32 experts_met(const b200moe_shape& s, u64 slots, u32 max_union) {
    const double of = slots > max_union ? max_union : s.experts;
    const double none = std::pow(1.0 - static_cast<double>(s.top_k) / s.experts, static_cast<double>(slots) / s.top_k);  // of its rows, whose experts are distinct, choose one
    return std::min(max_union, static_cast<u32>(std::ceil(of * (1.0 - none) - 1e-6)));
}

namespace {

constexpr u32 kMaxExperts = 1024, kMaxTopK = 32;

struct Carver {  // caller-owned workspace, 256-byte aligned sections
    unsigned char* base;
    u64 used = 0;
    explicit Carver(void* p) : base(static_cast<unsigned char*>(p)) {}
    template <class T>
    T* take(u64 count) {
        used = (used + 255) & ~u64(255);
        T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
        used += count * sizeof(T);
        return p;
    }
};

int check_shape(const b200moe_shape& s) {
    B200_REQUIRE(is_ds41_type(s.gate_type) || is_kquant(s.gate_type), "gate/up type %u is not bound (Q8_0 = 8, Q2_K = 10, Q4_K = 12, Q5_K = 13)", s.gate_type);
    B200_REQUIRE(is_ds41_type(s.down_type) || s.down_type == B200MOE_TYPE_Q4_K || s.down_type == B200MOE_TYPE_Q5_1,
                 "down type %u is not bound (Q5_1 = 7, Q8_0 = 8, Q2_K = 10, Q4_K = 12)", s.down_type);
    B200_REQUIRE(!(is_ds41_type(s.gate_type) && !is_ds41_type(s.down_type)), "Q8_0 / Q2_K gate/up with a down type other than Q8_0 / Q2_K has no declared contract");
    B200_REQUIRE(!(is_kquant(s.gate_type) && s.down_type == B200MOE_TYPE_Q2_K), "Q2_K down tensors belong to the Q8_0 / Q2_K family");
    B200_REQUIRE(s.hidden && s.inter && s.experts && s.top_k, "shape has a zero dimension");
    B200_REQUIRE(s.experts <= kMaxExperts && s.top_k <= kMaxTopK && s.top_k <= s.experts, "need top_k <= 32, top_k <= experts <= 1024");
    B200_REQUIRE(s.hidden % ((is_kquant(s.gate_type) || s.gate_type == B200MOE_TYPE_Q2_K) ? 256u : 32u) == 0, "hidden %u is not a whole number of gate/up blocks", s.hidden);
    B200_REQUIRE(s.inter % ((s.down_type == B200MOE_TYPE_Q4_K || s.down_type == B200MOE_TYPE_Q2_K) ? 256u : 32u) == 0, "inter %u is not a whole number of down blocks", s.inter);
    B200_REQUIRE(s.hidden % 64 == 0, "hidden %u must be a multiple of 64", s.hidden);
    return B200MOE_OK;
}
int check_a8(const b200moe_a8_rows& a, u32 rows, u32 width, bool need_sums, const char* what) {
    const u32 stride = a.stride ? a.stride : a.width;
    B200_REQUIRE(a.codes && a.deltas, "%s: A8 codes / deltas are null", what);
    B200_REQUIRE(!need_sums || a.sums, "%s: A8 sums are required by this contract", what);
    B200_REQUIRE(a.width == width && stride >= width && stride % 32 == 0, "%s: A8 width %u / stride %u do not fit width %u", what, a.width, stride, width);
    B200_REQUIRE(a.rows >= rows, "%s: A8 view holds %u rows, %u needed", what, a.rows, rows);
    B200_REQUIRE(aligned(a.codes, 16) && aligned(a.deltas, 8) && (!a.sums || aligned(a.sums, 8)), "%s: A8 pointers must be 16 / 8-byte aligned", what);
    return B200MOE_OK;
}
int check_routes(const b200moe_routes& r) {
    B200_REQUIRE(r.experts && r.begins && r.rows && r.slots && r.counts, "routes arrays are null");
    return B200MOE_OK;
}
int check_policy(const b200moe_route_policy& p) {
    B200_REQUIRE(p.experts && p.top_k && p.top_k <= p.experts, "route policy: need 0 < top_k <= experts");
    B200_REQUIRE(p.experts <= kMaxExperts && p.top_k <= kMaxTopK, "route policy: experts <= 1024 and top_k <= 32");
    B200_REQUIRE(p.score <= B200MOE_SCORE_SQRT_SOFTPLUS && p.key <= B200MOE_KEY_ORDERED_BITS && p.order <= B200MOE_ORDER_ASCENDING_ID, "route policy: unknown enum value");
    B200_REQUIRE(p.n_group >= 1 && p.topk_group >= 1 && p.topk_group <= p.n_group, "route policy: need 1 <= topk_group <= n_group");
    if (p.n_group > 1) {
        B200_REQUIRE(p.n_group <= 32 && p.experts % p.n_group == 0, "route policy: n_group must divide experts and be <= 32");
        B200_REQUIRE(p.experts / p.n_group >= 2 && u64(p.topk_group) * (p.experts / p.n_group) >= p.top_k, "route policy: the kept groups hold fewer than top_k experts");
    }
    return B200MOE_OK;
}

struct LayerScratch {
    b200moe_routes routes;
    u32* routes_scratch;
    b200moe_a8_rows act;
    float* raw;
    u32* summary;
    u32* row_status;
    u32* aux;  // [capacity * top_k] words for callers of the layer pieces
    u64 bytes;
};
LayerScratch carve_layer(void* ws, const b200moe_shape& s, u32 capacity) {
    Carver c(ws);
    const u64 n = u64(capacity) * s.top_k;
    LayerScratch L{};
    L.routes.experts = c.take<u32>(n);
    L.routes.begins = c.take<u32>(n + 1);
    L.routes.rows = c.take<u32>(n);
    L.routes.slots = c.take<u32>(n);
    L.routes.order = c.take<u32>(n);
    L.routes.low_counts = c.take<u32>(capacity);
    L.routes.counts = c.take<u32>(4);
    L.routes_scratch = c.take<u32>(routes_scratch_words(capacity, s.top_k, s.experts));
    L.act.codes = c.take<i8>(n * s.inter);
    L.act.deltas = c.take<float>(n * (s.inter / 32));
    L.act.sums = c.take<i32>(n * (s.inter / 32));
    L.act.rows = static_cast<u32>(n); L.act.width = s.inter; L.act.stride = s.inter;
    L.raw = c.take<float>(n * s.hidden);
    L.summary = c.take<u32>(4);
    L.row_status = c.take<u32>(capacity);
    L.aux = c.take<u32>(n);
    L.bytes = (c.used + 255) & ~u64(255);
    return L;
}

struct FfnScratch {
    b200moe_a8_rows x;
    float* logits;
    u32* ids;
    float* weights;
    void* x_dev;
    float* y_dev;
    float* x_f32;  // bfloat16 activations widened for the router
    void* layer;
    u64 bytes;
};
FfnScratch carve_ffn(void* ws, const b200moe_shape& s, u32 capacity) {
    Carver c(ws);
    FfnScratch F{};
    F.x.codes = c.take<i8>(u64(capacity) * s.hidden);
    F.x.deltas = c.take<float>(u64(capacity) * (s.hidden / 32));
    F.x.sums = c.take<i32>(u64(capacity) * (s.hidden / 32));
    F.x.rows = capacity; F.x.width = s.hidden; F.x.stride = s.hidden;
    F.logits = c.take<float>(u64(capacity) * s.experts);
    F.ids = c.take<u32>(u64(capacity) * s.top_k);
    F.weights = c.take<float>(u64(capacity) * s.top_k);
    F.x_dev = c.take<float>(u64(capacity) * s.hidden);
    F.y_dev = c.take<float>(u64(capacity) * s.hidden);
    F.x_f32 = c.take<float>(u64(capacity) * s.hidden);
    const u64 at = (c.used + 255) & ~u64(255);
    F.layer = ws ? static_cast<unsigned char*>(ws) + at : nullptr;
    F.bytes = at + carve_layer(nullptr, s, capacity).bytes;
    return F;
}

// The status words that a call owns: the job summary and, where the caller gives none of his own, the rows' status. They are cleared by the launch that
// builds the routes (a caller's summary word too): a memset node in front of it cost 3 us of a short call.
RoutesClear clear_of(const LayerScratch& L, u32* caller_row_status, u32* caller_summary) {
    return RoutesClear{caller_row_status ? nullptr : L.row_status, L.summary, caller_summary};
}

// What a window is for the kernels that walk it item by item, known from its sizes alone: the items of eight entries and the tiles of 32 that
// its experts make when the entries are spread evenly (the last item of an expert is half full on average, and an expert has one tile until it has
// about 20 entries), and whether a tile has 16 entries at most.
struct Window { u64 items8, tiles32; bool few; };
Window window_of(const b200moe_shape& s, u32 rows, u32 max_union) {
    if (s.experts == 1) return Window{(u64(rows) + 7) / 8, (u64(rows) + 31) / 32, rows <= 16};
    const u64 e16 = 16 * u64(rows) * s.top_k / s.experts;  // entries an expert, in sixteenths
    return Window{(max_union * std::max<u64>(16, e16 / 8 + 7) + 15) / 16, (max_union * std::max<u64>(16, (e16 + 192) / 32) + 15) / 16, e16 <= 12 * 16};
}
u64 waves(u64 items, u64 at_once) { return (items + at_once - 1) / at_once; }
// Plan by window size, chosen on the host from the sizes (no environment reads inside numerical code): decode
// windows of Q4_K experts take the persistent bulk-copy forms, prompts the grouped form.
// grouped_min_rows: windows of at least that many rows take the grouped form; 0 = chosen here, for gate/up and down each.
// Where the segment-streaming form applies, the grouped one (tiles of 32 entries) takes over from it (items of 8) where its waves take less time,
// both by their sizes: a tile 2 us + 1.75 a super-block of its rows; an item 1.38 us + 0.46 a super-block (1.7 + 0.56 where rows have less than three and a
// stage holds one), two an SM, or 0.4 a super-block where there are no more items than SMs. Whole calls with both launches in the streaming and in the
// grouped form, us: 128 experts of 2048 x 768, top-8, 143 and 200 with 128 rows, 190 and 212 with 192, 213 and 219 with 224, 234 and 225 with 256; 64 of 7168 x 2048,
// top-8, 470 and 775 with 64 rows, 638 and 765 with 96, 718 and 785 with 112, 802 and 818 with 128 (781 with gate/up grouped); 16 of 4096 x 1536, top-2, 123 and 140 with 128,
// 165 and 142 with 200; one expert of 5120 x 17408 108 and 215 with 24 rows, 158 and 216 with 32, 180 and 252 with 40 (197 with gate/up grouped), 213 and 255 with 56 (197),
// 265 and 257 with 64 (229). The estimates of the waves lie within 10 % of these. Below 32 rows they have not been followed, below 48 only where they see more than a few
// percent gained. Layers with a down of other blocks, gate/up in either form: 64 of 2560 x 768, top-4, 262 and 274 with 204 rows, 449 and 424 with 400.
// Where the segment-streaming form does not apply (more than 8192 slots, rows that bulk copies cannot take) the alternative is the
// per-block form, and 128 rows are the line.
constexpr u32 kGroupedLeastRows = 32, kGroupedSureRows = 48, kGroupedRowsElse = 128;
bool grouped_pays(const b200moe_shape& s, u32 rows, u32 max_union, u32 grouped_min_rows, bool streams, bool down) {
    if (grouped_min_rows) return rows >= grouped_min_rows;
    if (!streams) return rows >= kGroupedRowsElse;
    if (rows < kGroupedLeastRows) return false;
    const Window w = window_of(s, rows, max_union);
    const u64 blocks = (down ? s.inter : s.hidden) / 256, sms = static_cast<u64>(device_sm_count());
    const u64 items = w.items8 * (down ? s.hidden / 64 : s.inter / 32), item = blocks < 3 ? 1700 + 560 * blocks : 1375 + 460 * blocks;  // ns
    const u64 streaming = items <= sms ? std::min<u64>(item, 1375 + 400 * blocks) : waves(items, 2 * sms) * item;
    const u64 grouped = waves(w.tiles32 * grouped_row_tiles(down ? s.hidden : s.inter, down), sms) * (2000 + 1750 * blocks);
    return grouped * (rows < kGroupedSureRows ? 107 : 100) < streaming * 100;
}
// The other forms of the Q4_K GEMVs: the segment-streaming form (any row length; its items are dealt out dynamically) wherever it applies, else the
// row-streaming form (a ring of whole rows, its work split fixed per CTA) and the per-block form. In a call the segment-streaming form has windows of one
// and two rows too, since it begins its launches with the weights of its first items. Whole calls, row and segment streaming, us: 128
// experts of 2048 x 768, one row, top 1 to 16, 30.8 and 28.7, 32.9 and 30.8, 36.9 and 34.7 (top 8), 45.1 and 41.2; two rows, top 8, 43.0 and 39.2; 16
// experts of 512 x 256 28.7 and 26.6; dense 2048 x 2048 23.7 and 17.5, 512 x 512 21.5 and 15.4. B200MOE_DEBUG_DECODE_FORM forces
// one of the four where it applies, whatever grouped_min_rows says.
// Stages called by themselves (alone: nothing is known of the launch in front, so none starts early) keep the row-streaming form for one row of up to 2048
// weights and, where rows are short, for two. A launch, us, row and segment streaming: gate/up of 64 of 2048 x 768, top-4, 6.8 and 7.8 with 1 row, 8.2 and 9.4
// with 2; down 5.6 and 6.4, 7.3 and 6.7; down of 128 of 1024 x 256, top-8, 4.9 and 6.4, 5.7 and 6.5. Inside a layer gate/up is better off in the segment-streaming
// form too (a call over 128 experts of 2048 x 768, one row, top 8, 24.0 and 23.5).
bool row_stream_alone(u32 rows, u32 K, bool down) { return rows <= 1 ? K <= 2048 : rows == 2 && K <= (down ? 512u : 2048u); }
enum class Q4Form { grouped, row_stream, wide, block };
Q4Form pick_q4_form(const b200moe_shape& s, bool grouped_fits, bool row_stream_fits, bool wide_fits, u32 rows, u32 max_union, u32 grouped_min_rows, bool alone, bool down) {
    const u32 forced = debug_value(B200MOE_DEBUG_DECODE_FORM);
    if (forced == 1 && row_stream_fits) return Q4Form::row_stream;
    if (forced == 2 && wide_fits) return Q4Form::wide;
    if (forced == 3) return Q4Form::block;
    if (forced == 5 && grouped_fits) return Q4Form::grouped;
    if (grouped_fits && grouped_pays(s, rows, max_union, grouped_min_rows, wide_fits, down)) return Q4Form::grouped;
    if (row_stream_fits && alone && row_stream_alone(rows, down ? s.inter : s.hidden, down)) return Q4Form::row_stream;
    if (wide_fits) return Q4Form::wide;
    return row_stream_fits ? Q4Form::row_stream : Q4Form::block;
}
// The DS41 family (Q8_0 x A8). Below kFewRows rows: a CTA one item with all its weights asked for at once (gemv_q8_shot.cu, rows of whole units of 256
// weights), else one weight row per warp. From there on the tensor-core form of gemv_q8_mma.cu (rows of 1024 to 7168 weights), else the dp4a token-block form of
// gemv_q8_wide.cu. The one-item form pays by the entry and keeps a multiprocessor for one item, so it gives way to the tensor-core form early where an expert has
// more than four entries of long rows. From 8 rows on it is the better one only in windows so sparse that an expert has an entry at most, against the tensor-core
// form, for down and for few items of gate/up (14 runs of 32 blocks a multiprocessor). Whole calls, one-item and tensor-core form, us: one expert of
// 7168 x 2048 45 and 53 with 1 row, 55 and 56 with 4, 59 and 57 with 5, 64 and 59 with 7; of 2048 x 1024 31 and 37, 35 and 37 with 4, 37 and 39 with 6,
// 39 and 38 with 7; 64 of 2048 x 1024, top-4, 80 and 81 with 7 rows; 16 of 4096 x 1536, top-2, 61 and 64 with 4, 82 and 80 with 6, 86 and 82 with 8.
// Layers, both stages in the tensor-core form, down alone and both in the one-item form: 64 of 2048 x 1024, top-4, 68.4, 63.9 and 67.0 with 8 rows, 93.2, 88.7
// and 91.3 with 12; 512 of 1024 x 1024, top-4, 79.4, 74.2 and 69.1 with 12, 157.7, 151.6 and 156.1 with 32. Against the token-block form down loses: 256 of 2048 x 768,
// top-8, 96.7 and 109.9 with 8 rows, 202 and 249 with 24.
// The grouped form (grouped_q8.cu, tiles of 32 entries) takes over from the tensor-core form where its waves of tiles take less time than the
// other's waves of items, both by their sizes: a tile 2.3 us + 0.7 a unit of 256 columns with up to 16 entries, 2.6 + 0.77 with more, an item of
// 32 gate and up rows 3 us + 0.33 a unit, one of 32 down rows half of that. Tensor-core and grouped form, gate/up and down: one expert of
// 2048 x 17408 28.8 and 32.3 us with 8 rows, 51.4 and 32.9 with 16, 72 and 39 with 20; of 7168 x 2048 18.6 and 22.8, 16.5 and 12.4 with 16 rows; of
// 1024 x 1024 8.4 and 10.3 (down) with 20; four of 2048 x 4096, top-2, 45 and 33, 22 and 16.6 with 20 rows; 64 of 2048 x 1024, top-4, whole
// calls, 180 and 196 with 80 rows, 183 and 197 with 96, 207 and 198 with 112, 230 and 200 with 128; 16 of 4096 x 1536, top-2, 69 and 74, 53 and 43 with 64. Where the tensor-core form does not apply (rows below
// 1024 or above 7168 weights) the grouped one takes over from the dp4a form at 4 entries an expert: down of 48 experts of 2048 x 512 36.8 and 39 us with 3,
// 41 and 38.5 with 4, 49 and 39 with 5; of 32 of 1536 x 768 29 and 28 with 4.5; one expert of 2048 x 17408 45 and 43 us with 8 rows, 53.4 and 53.5 with
// 17, of 4096 x 12288 35 and 33 with 8, 84 and 40 with 24.
constexpr u32 kFewRows = 8;
enum class Q8Form { row_per_warp, shot, wide, mma, grouped };
bool q8_grouped_pays(const b200moe_shape& s, bool mma_fits, u32 rows, u32 max_union, bool down) {
    if (rows < kFewRows) return false;
    if (!mma_fits) return u64(rows) * s.top_k >= u64(4) * s.experts;
    const Window w = window_of(s, rows, max_union);
    const u64 units = (down ? s.inter : s.hidden) / 256, sms = static_cast<u64>(device_sm_count());
    const u64 tile = w.few ? 2300 + 700 * units : 2600 + 770 * units, item = (3000 + 330 * units) / (down ? 2 : 1);  // ns
    const u64 grouped = waves(w.tiles32 * (down ? s.hidden / 64 : s.inter / 32), sms) * tile, tensor = waves(w.items8 * ((down ? s.hidden : s.inter) / 32), sms) * item;
    return grouped < tensor;
}
Q8Form pick_q8_form(const b200moe_shape& s, bool shot_fits, bool wide_fits, bool mma_fits, bool grouped_fits, u32 rows, u32 max_union, bool down) {
    const u32 forced = debug_value(B200MOE_DEBUG_DECODE_FORM);
    if (forced == 3) return Q8Form::row_per_warp;
    if (grouped_fits && (forced == 5 || (forced == 0 && q8_grouped_pays(s, mma_fits, rows, max_union, down)))) return Q8Form::grouped;
    if (forced == 4 && mma_fits) return Q8Form::mma;
    if (forced == 2 && wide_fits) return Q8Form::wide;
    if (forced == 6 && shot_fits) return Q8Form::shot;
    if (forced == 0) {
        const u64 slots = u64(rows) * s.top_k;
        const u32 longest = std::max(s.hidden, s.inter);
        const bool sparse = mma_fits && longest <= 2048 && 4 * slots <= u64(3) * s.experts;
        const u64 runs = slots * (s.inter / 32) * ((s.hidden + 1023) / 1024);  // that a sparse window's gate/up brings in, each 32 blocks of 64 rows
        const bool shot = rows < kFewRows ? longest <= 2048 || slots <= u64(4) * s.experts || !mma_fits : sparse && (down || runs <= u64(14) * static_cast<u32>(device_sm_count()));
        if (shot_fits && shot) return Q8Form::shot;
        if (mma_fits && (rows >= kFewRows || shot_fits)) return Q8Form::mma;
        if (wide_fits && rows >= kFewRows) return Q8Form::wide;
    }
    return Q8Form::row_per_warp;
}
// The four-chain down on the tensor cores (down_chain4_mma.cu), else in the dp4a forms of gemv_q4k.cu. By the entries of an expert: slots over ALL experts, since of a rank's share
// of the experts the window's slots are a share too. The dp4a forms pay by the entry, and the more the longer the rows, so the line falls with their length: from 3.5 (Q8_0) and 4.5
// entries (Q5_1) at 128 weights to none and one at 1024. A window whose items are no more than SMs is one item's time and has the tensor cores from a
// quarter of an entry on (below, a share of the experts often has none, and a launch without items takes 1.2 us longer there). Layers, us, the better
// dp4a form and this: 128 experts of 640 -> 2560, top 8, Q5_1 16 rows 74.0 and 85.9, 40 115.5 and 121.4, 48 127.0 and 129.4, 64 151.8 and 139.9, a quarter of them owned 31.3 and
// 35.3, 43.6 and 41.5, 44.2 and 41.8, 56.2 and 48.7; Q8_0 24 rows 104 and 114, 32 119 and 121, 48 146 and 138, a quarter owned 40.4 and 39.5, 48.4 and 46.8, 53.3 and 48.2; 60 of
// 768 -> 2560, top 4, Q5_1 15 rows 48.3 and 53.2, 30 74.7 and 73.2, 45 86.6 and 78.4, Q8_0 8 rows 40.0 and 42.3, 15 52.3 and 51.5, 30 78.9 and 67.0; of 1536 -> 2560 Q5_1 8 rows
// 64.0 and 68.9, 15 91.3 and 95.8, 60 176 and 147, Q8_0 1 row 20.0 and 19.5, 15 115 and 81; 128 of 128 -> 1024, top 8, 40 rows 30.9 and 37.8, 30.3 and 38.0, 80 38.6 and 41.1, 37.8 and
// 41.2; one wave: 16 of 640 -> 512, top 2, 3 rows 13.1 and 12.6, 13.3 and 12.9, 8 of 64 of 512 -> 1024, top 4, 24 rows 15.8 and 14.3, 16.5 and 14.3. Over 1500 random layers (1 to
// 256 experts, all or a half to an eighth of them owned, 128 to 2048 wide, 0.1 to 12 entries an expert) the choice lies 0.6 % above the best form's time.
// A stage called by itself cannot ask for weights ahead, which the tensor-core form lives on more: the line lies 256 weights further, and 24 entries or fewer keep the dp4a forms
// (16 of 640 -> 512, top 2, 3 rows, a launch, 3.7 and 4.3). So do Q5_1 rows of up to 1024 weights with 256 entries or fewer, where they are the slower ones (32 of 1024 -> 2048, top 4,
// 64 rows 57 and 26): the line between the two dp4a forms is held by calls of that size.
bool chain4_mma_pays(const b200moe_down_view& v, u64 slots, bool alone, u32 chunks) {
    const b200moe_shape& s = v.shape;
    const bool q51 = s.down_type == B200MOE_TYPE_Q5_1;
    if (alone && slots <= (q51 && s.inter <= 1024 ? 256u : 24u)) return false;
    if (!alone && slots * 4 >= s.experts && u64(experts_met(s, slots, v.max_union)) * chunks <= static_cast<u32>(device_sm_count())) return true;
    const u32 none = (q51 ? 1280u : 1024u) + (alone ? 256u : 0u), least = std::max(q51 ? 256u : 0u, none - std::min(none, s.inter));  // in 256ths of an entry
    return slots * 256 > u64(s.experts) * least;
}
int enqueue_gate_up(const b200moe_gate_up_view& v, u32 rows, cudaStream_t st, u32 grouped_min_rows = 0, const ChainHints& hints = {}) {
    if (v.shape.gate_type == B200MOE_TYPE_Q2_K) return launch_gate_up_ds41_any(v, st);  // the generic form of the family reads every block type
    if (!is_kquant(v.shape.gate_type)) {
        switch (pick_q8_form(v.shape, q8_shot_gate_up_fits(v, rows), q8_wide_gate_up_fits(v, rows), q8_mma_gate_up_fits(v, rows), grouped_q8_gate_up_fits(v), rows, v.max_union, false)) {
            case Q8Form::shot: return launch_gate_up_q8_shot(v, rows, hints, st);
            case Q8Form::grouped: return launch_gate_up_q8_grouped(v, st);
            case Q8Form::mma: return launch_gate_up_q8_mma(v, rows, st);
            case Q8Form::wide: return launch_gate_up_q8_wide(v, rows, st);
            default: return launch_gate_up_q8(v, st);
        }
    }
    // Q5_K: the segment-streaming and the per-block form read both K-quant layouts. The first wherever it fits; us a layer call, per-block form and this: 1 row of 2560 -> 768
    // 36.2 and 27.2 (1024 -> 512: 22.8 and 21.8), 24 rows of 2560 -> 1024 228 and 120, 100 rows of 2560 -> 768 457 and 166, 400 rows of 2048 -> 544 1697 and 589.
    if (v.shape.gate_type == B200MOE_TYPE_Q5_K) {
        const u32 forced = debug_value(B200MOE_DEBUG_DECODE_FORM);
        return (forced == 0 || forced == 2) && wide_gate_up_fits(v, rows) ? launch_gate_up_q4k_wide(v, rows, hints, st) : launch_gate_up_q4k(v, st);
    }
    switch (pick_q4_form(v.shape, grouped_gate_up_fits(v), stream_gate_up_fits(v, rows), wide_gate_up_fits(v, rows), rows, v.max_union, grouped_min_rows, hints.slots == 0, false)) {
        case Q4Form::grouped: return launch_gate_up_q4k_grouped(v, st);
        case Q4Form::row_stream: return launch_gate_up_q4k_stream(v, rows, st);
        case Q4Form::wide: return launch_gate_up_q4k_wide(v, rows, hints, st);
        default: return launch_gate_up_q4k(v, st);
    }
}
int enqueue_down(const b200moe_down_view& v, u32 rows, cudaStream_t st, u32 grouped_min_rows = 0, const ChainHints& hints = {}) {
    if (v.shape.down_type == B200MOE_TYPE_Q4_K) {
        switch (pick_q4_form(v.shape, grouped_down_fits(v), stream_down_fits(v, rows), wide_down_fits(v, rows), rows, v.max_union, grouped_min_rows, hints.slots == 0, true)) {
            case Q4Form::grouped: return launch_down_q4k_grouped(v, st);
            case Q4Form::row_stream: return launch_down_q4k_stream(v, rows, st);
            case Q4Form::wide: return launch_down_q4k_wide(v, rows, hints, st);
            default: return launch_down_q4k(v, st);
        }
    }
    if (is_kquant(v.shape.gate_type)) {  // chain4: Q8_0 and Q5_1 blocks
        const u32 forced = debug_value(B200MOE_DEBUG_DECODE_FORM);
        const u32 chunks = forced == 0 || forced == 5 ? chain4_mma_chunks(v) : 0u;
        if (chunks && (forced == 5 || chain4_mma_pays(v, u64(rows) * v.shape.top_k, hints.slots == 0, chunks))) return launch_down_chain4_mma(v, hints, st);
        return launch_down_q8_chain4(v, rows, hints, st);
    }
    if (v.shape.down_type == B200MOE_TYPE_Q2_K) return launch_down_ds41_any(v, st);
    switch (pick_q8_form(v.shape, q8_shot_down_fits(v, rows), q8_wide_down_fits(v, rows), q8_mma_down_fits(v, rows), grouped_q8_down_fits(v), rows, v.max_union, true)) {
        case Q8Form::shot: return launch_down_q8_shot(v, rows, hints, st);
        case Q8Form::grouped: return launch_down_q8_grouped(v, st);
        case Q8Form::mma: return launch_down_q8_mma(v, rows, st);
        case Q8Form::wide: return launch_down_q8_wide(v, rows, st);
        default: return launch_down_q8(v, hints, st);
    }
}

}  // namespace
}  // namespace b200moe

using namespace b200moe;

extern "C" {

int b200moe_abi_version(void) { return B200MOE_ABI_VERSION; }
const char* b200moe_last_error(void) { return last_error_slot().c_str(); }
const char* b200moe_last_launch(void) { return last_launch_slot(); }
uint64_t b200moe_launch_count(void) { return launch_counter().load(std::memory_order_relaxed); }
int b200moe_debug_set(uint32_t key, uint32_t value) {
    B200_REQUIRE(key < 3, "debug_set: unknown key %u", key);
    g_debug[key].store(value, std::memory_order_relaxed);
    return B200MOE_OK;
}

uint64_t b200moe_gate_row_bytes(const b200moe_shape* s) { return s ? row_bytes_of(s->gate_type, s->hidden) : 0; }
uint64_t b200moe_down_row_bytes(const b200moe_shape* s) { return s ? row_bytes_of(s->down_type, s->inter) : 0; }
uint64_t b200moe_expert_bytes(const b200moe_shape* s) {
    return s ? 2 * row_bytes_of(s->gate_type, s->hidden) * s->inter + row_bytes_of(s->down_type, s->inter) * s->hidden : 0;
}

int b200moe_quantize_a8(const b200moe_quantize_a8_view* v, void* stream) {
    B200_REQUIRE(v, "null view");
    B200_REQUIRE(v->width % 32 == 0, "A8 activation width must be a multiple of 32 (got %u)", v->width);
    if (v->rows == 0 || v->width == 0) return B200MOE_OK;
    B200_REQUIRE(v->x, "quantize_a8: x is null");
    const u32 xs = v->x_stride ? v->x_stride : v->width;
    B200_REQUIRE(xs >= v->width, "quantize_a8: x_stride %u is below the width %u", xs, v->width);
    const u32 stride = v->out.stride ? v->out.stride : v->out.width;
    B200_REQUIRE(v->out.codes && v->out.deltas, "quantize_a8: output codes / deltas are null");
    B200_REQUIRE(v->out.width == v->width && stride >= v->width && stride % 32 == 0 && v->out.rows >= v->rows, "quantize_a8: output view does not fit rows %u x width %u", v->rows, v->width);
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return launch_quantize_a8(*v, as_stream(stream));
}

int b200moe_rmsnorm_a8(const b200moe_rmsnorm_view* v, void* stream) {
    B200_REQUIRE(v, "null view");
    B200_REQUIRE(v->n % 32 == 0, "rmsnorm: n must be a multiple of 32 (got %u)", v->n);
    if (v->rows == 0 || v->n == 0) return B200MOE_OK;
    B200_REQUIRE(v->x, "rmsnorm: x is null");
    B200_REQUIRE(v->out || v->a8.codes, "rmsnorm: neither out nor a8 is given");
    const u32 xs = v->x_stride ? v->x_stride : v->n, os = v->out_stride ? v->out_stride : v->n;
    B200_REQUIRE(xs >= v->n && os >= v->n, "rmsnorm: a stride is below n = %u", v->n);
    if (v->a8.codes) {
        const u32 stride = v->a8.stride ? v->a8.stride : v->a8.width;
        B200_REQUIRE(v->a8.deltas, "rmsnorm: a8.deltas is null");
        B200_REQUIRE(v->a8.width == v->n && stride >= v->n && stride % 32 == 0 && v->a8.rows >= v->rows, "rmsnorm: a8 view does not fit rows %u x n %u", v->rows, v->n);
    }
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return launch_rmsnorm_a8(*v, as_stream(stream));
}

int b200moe_q8_0_a8(const b200moe_q8a8_view* v, void* stream) {
    B200_REQUIRE(v, "null view");
    B200_REQUIRE(v->width % 32 == 0, "Q8_0 product width must be a multiple of 32 (got %u)", v->width);
    if (v->count == 0 || v->x.rows == 0 || v->width == 0) return B200MOE_OK;
    B200_REQUIRE(v->weight && v->out, "q8_0_a8: weight / out are null");
    B200_REQUIRE(v->row_bytes >= v->width / 32 * kQ8Block, "q8_0_a8: row_bytes %u is below %u", v->row_bytes, v->width / 32 * kQ8Block);
    if (int rc = check_a8(v->x, v->x.rows, v->width, false, "q8_0_a8 x")) return rc;
    const u32 os = v->out_stride ? v->out_stride : v->count;
    B200_REQUIRE(os >= v->count, "q8_0_a8: out_stride %u is below count %u", os, v->count);
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return launch_q8_0_a8(*v, as_stream(stream));
}

int b200moe_router(const b200moe_router_view* v, void* stream) {
    B200_REQUIRE(v, "null view");
    if (int rc = check_policy(v->policy)) return rc;
    B200_REQUIRE(v->logits && v->ids && v->weights, "router: logits / ids / weights are null");
    B200_REQUIRE(!v->policy.selection_bias || v->bias, "router: the policy has a selection bias but bias is null");
    if (v->x) {
        B200_REQUIRE(v->weight && v->hidden, "router: weight is null or hidden is 0");
        const u32 xs = v->x_stride ? v->x_stride : v->hidden;
        B200_REQUIRE(xs >= v->hidden, "router: x_stride %u is below hidden %u", xs, v->hidden);
    }
    if (v->rows == 0) return B200MOE_OK;
    if (!device_ready()) return B200MOE_ERR_CUDA;
    if (v->x) if (int rc = launch_router_logits(*v, as_stream(stream))) return rc;
    return launch_router_select(*v, as_stream(stream));
}

uint64_t b200moe_routes_scratch_words(uint32_t rows, uint32_t top_k, uint32_t experts) { return routes_scratch_words(rows, top_k, experts); }

}  // extern "C"
namespace b200moe {
int b200moe_check_routes_view(const b200moe_routes_view* v) {
    B200_REQUIRE(v, "null view");
    B200_REQUIRE(v->rows && v->top_k && v->ids, "routes need rows * top_k expert ids");
    B200_REQUIRE(v->experts && v->experts <= kMaxExperts && v->top_k <= kMaxTopK && v->top_k <= v->experts, "routes: need top_k <= 32, top_k <= experts <= 1024");
    B200_REQUIRE(v->end <= v->experts && (v->end == 0 || v->first < v->end) && v->base <= v->first, "routes: expert range [%u, %u) base %u is inconsistent", v->first, v->end, v->base);
    if (int rc = check_routes(v->out)) return rc;
    B200_REQUIRE(v->out.order && v->out.low_counts, "routes: order / low_counts are null");
    B200_REQUIRE(u64(v->rows) * v->top_k <= 1024 || v->scratch, "routes: more than 1024 slots need scratch");
    return B200MOE_OK;
}
}  // namespace b200moe
extern "C" {

int b200moe_build_routes(const b200moe_routes_view* v, void* stream) {
    if (int rc = b200moe_check_routes_view(v)) return rc;
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return launch_routes(*v, RoutesClear{}, as_stream(stream));
}

int b200moe_gate_up(const b200moe_gate_up_view* v, void* stream) {
    B200_REQUIRE(v, "null view");
    if (int rc = check_shape(v->shape)) return rc;
    if (int rc = check_routes(v->routes)) return rc;
    B200_REQUIRE(v->weights.gate && v->weights.up && aligned(v->weights.gate, 16) && aligned(v->weights.up, 16), "gate_up: gate / up tensors must be non-null and 16-byte aligned");
    B200_REQUIRE((v->gate_out == nullptr) == (v->up_out == nullptr), "gate_up: gate_out and up_out come together");
    const bool q4k = is_kquant(v->shape.gate_type);
    if (int rc = check_a8(v->x, 0, v->shape.hidden, q4k, "gate_up x")) return rc;
    if (int rc = check_a8(v->act, 0, v->shape.inter, down_reads_sums(v->shape.down_type), "gate_up act")) return rc;
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return enqueue_gate_up(*v, v->x.rows, as_stream(stream));
}

int b200moe_down(const b200moe_down_view* v, void* stream) {
    B200_REQUIRE(v, "null view");
    if (int rc = check_shape(v->shape)) return rc;
    if (int rc = check_routes(v->routes)) return rc;
    B200_REQUIRE(v->weights.down && aligned(v->weights.down, 16) && v->raw, "down: the down tensor must be non-null and 16-byte aligned, raw non-null");
    if (int rc = check_a8(v->act, 0, v->shape.inter, down_reads_sums(v->shape.down_type), "down act")) return rc;
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return enqueue_down(*v, v->act.rows / v->shape.top_k, as_stream(stream));
}

int b200moe_combine(const b200moe_combine_view* v, void* stream) {
    B200_REQUIRE(v, "null view");
    B200_REQUIRE(v->raw && v->weights && (v->y || v->y_blocks), "combine: raw / weights / y are null");
    B200_REQUIRE(!v->y_blocks || (v->y_block_rows && !v->y_bf16), "combine: y_blocks needs y_block_rows > 0 and no y_bf16");
    B200_REQUIRE(v->top_k && v->top_k <= kMaxTopK && v->hidden, "combine: need 0 < top_k <= 32 and hidden > 0");
    B200_REQUIRE(v->form <= B200MOE_COMBINE_FMA_SLOTS, "combine: unknown form %u", v->form);
    if (v->form == B200MOE_COMBINE_PARTS) {
        B200_REQUIRE((v->ids || v->low_counts) && v->order, "combine(parts): ids (or low_counts) / order are null");
        B200_REQUIRE(!v->low_counts || v->parts == 2, "combine(parts): low_counts describes a two-part split (parts must be 2)");
        B200_REQUIRE(v->parts && (v->part_experts || v->low_counts) && v->only_part < static_cast<int>(v->parts), "combine(parts): parts / part_experts / only_part are inconsistent");
        B200_REQUIRE(v->only_part_count <= 1 || (v->only_part >= 0 && v->only_part + v->only_part_count <= v->parts && v->part_stride && !v->y_bf16),
                     "combine(parts): only_part_count needs only_part >= 0, a part_stride and no y_bf16");
    }
    if (v->rows == 0) return B200MOE_OK;
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return launch_combine(*v, as_stream(stream));
}

int b200moe_canonical_sum(const float* a, const float* b, const float* c, uint64_t count, float* y, void* stream) {
    B200_REQUIRE(a && b && y, "canonical_sum: a / b / y are null");
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return launch_canonical_sum(a, b, c, count, y, as_stream(stream));
}

uint64_t b200moe_layer_workspace_bytes(const b200moe_shape* s, uint32_t capacity) {
    if (!s || check_shape(*s)) return 0;
    return carve_layer(nullptr, *s, capacity).bytes;
}

static int layer_impl(const b200moe_layer_view* v, void* stream, bool routes_ready, bool fresh);
int b200moe_layer(const b200moe_layer_view* v, void* stream) { return layer_impl(v, stream, false, false); }
int b200moe_layer_fresh(const b200moe_layer_view* v, void* stream) { return layer_impl(v, stream, false, true); }

// routes_ready: the caller (b200moe_ffn) has already built the routes of v->ids into this workspace and cleared the
// status words (the fused select + routes launch of decode windows). fresh: rows that the call fails to write become zeros.
static int layer_impl(const b200moe_layer_view* v, void* stream, bool routes_ready, bool fresh) {
    B200_REQUIRE(v, "null view");
    if (int rc = check_shape(v->shape)) return rc;
    const b200moe_shape& s = v->shape;
    B200_REQUIRE(v->rows <= v->capacity, "layer: rows %u exceed the workspace capacity %u", v->rows, v->capacity);
    if (v->rows == 0) return B200MOE_OK;
    B200_REQUIRE(v->ids && v->route_weights, "layer: ids / route_weights are null");
    B200_REQUIRE(v->weights.gate && v->weights.up && v->weights.down, "layer: expert tensors are null");
    B200_REQUIRE(aligned(v->weights.gate, 16) && aligned(v->weights.up, 16) && aligned(v->weights.down, 16), "layer: expert tensors must be 16-byte aligned");
    if (int rc = check_a8(v->x, v->rows, s.hidden, is_kquant(s.gate_type), "layer x")) return rc;
    B200_REQUIRE(v->end <= s.experts && (v->end == 0 || v->first < v->end) && v->base <= v->first, "layer: expert range [%u, %u) base %u is inconsistent", v->first, v->end, v->base);
    B200_REQUIRE(v->combine_form <= B200MOE_COMBINE_FMA_SLOTS, "layer: unknown combine form %u", v->combine_form);
    if (v->y && v->combine_form == B200MOE_COMBINE_PARTS)
        B200_REQUIRE(v->parts && v->part_experts && v->only_part < static_cast<int>(v->parts), "layer: parts / part_experts / only_part are inconsistent");
    B200_REQUIRE(v->only_part_count <= 1 || (v->combine_form == B200MOE_COMBINE_PARTS && v->only_part >= 0 && v->only_part + v->only_part_count <= v->parts &&
                                             v->part_stride && !v->y_bf16),
                 "layer: only_part_count needs the PARTS form, only_part >= 0, a part_stride and no y_bf16");
    const LayerScratch L = carve_layer(v->workspace, s, v->capacity);
    if (!v->workspace || v->workspace_bytes < L.bytes)
        return fail(B200MOE_ERR_WORKSPACE, "layer: workspace of %llu bytes needed, %llu given", (unsigned long long)L.bytes, (unsigned long long)v->workspace_bytes);
    B200_REQUIRE(aligned(v->workspace, 256), "layer: workspace must be 256-byte aligned");
    if (!device_ready()) return B200MOE_ERR_CUDA;
    cudaStream_t st = as_stream(stream);

    u32* row_status = v->row_status ? v->row_status : L.row_status;
    u32* summary = v->summary ? v->summary : L.summary;

    b200moe_routes_view rv{};
    rv.ids = v->ids; rv.rows = v->rows; rv.top_k = s.top_k; rv.experts = s.experts;
    rv.split = v->part_experts ? v->part_experts : s.experts / 2;
    rv.first = v->first; rv.end = v->end; rv.base = v->base;
    rv.scratch = L.routes_scratch; rv.row_status = row_status; rv.out = L.routes;
    auto tap = [&](int i) {
        if (v->stage_events && v->stage_events[i]) cudaEventRecord(static_cast<cudaEvent_t>(v->stage_events[i]), st);
    };
    tap(0);
    if (!routes_ready) if (int rc = launch_routes(rv, clear_of(L, v->row_status, v->summary), st)) return rc;
    tap(1);

    const u32 span = (v->end ? v->end : s.experts) - v->first;
    const u32 max_union = static_cast<u32>(std::min<u64>(u64(v->rows) * s.top_k, span));
    float* raw = v->raw ? v->raw : L.raw;

    b200moe_gate_up_view gu{};
    gu.shape = s; gu.weights = v->weights; gu.routes = L.routes; gu.max_union = max_union;
    gu.x = v->x; gu.act = L.act; gu.row_status = row_status; gu.summary = summary;
    tap(2);
    const u64 slots = u64(v->rows) * s.top_k;
    if (int rc = enqueue_gate_up(gu, v->rows, st, v->grouped_min_rows, ChainHints{false, 0, slots})) return rc;
    tap(3);

    b200moe_down_view dn{};
    dn.shape = s; dn.weights = v->weights; dn.routes = L.routes; dn.max_union = max_union;
    dn.act = L.act; dn.raw = raw; dn.summary = summary;
    tap(4);
    if (int rc = enqueue_down(dn, v->rows, st, v->grouped_min_rows, ChainHints{true, 0, slots})) return rc;  // gate/up was admitted after the routes
    tap(5);

    if (!v->y && !v->y_blocks) return B200MOE_OK;
    B200_REQUIRE(!v->y_blocks || (v->y_block_rows && !v->y_bf16), "layer: y_blocks needs y_block_rows > 0 and no y_bf16");
    b200moe_combine_view cv{};
    cv.raw = raw; cv.shared = v->shared; cv.weights = v->route_weights; cv.ids = v->ids; cv.order = L.routes.order;
    cv.rows = v->rows; cv.top_k = s.top_k; cv.hidden = s.hidden; cv.form = v->combine_form;
    cv.parts = v->parts; cv.part_experts = v->part_experts; cv.only_part = v->only_part;
    cv.only_part_count = v->only_part_count; cv.part_stride = v->part_stride;
    cv.y = v->y; cv.y_bf16 = v->y_bf16; cv.y_blocks = v->y_blocks; cv.y_block_rows = v->y_block_rows;
    cv.row_status = is_kquant(s.gate_type) ? row_status : nullptr;
    cv.summary = summary;
    tap(6);
    // A projection that is not finite skips down for the whole job (any bit of the summary does), so raw holds an earlier call's values for the other rows
    // too: none is combined. Down was admitted after the routes; without an expert there was none.
    const int rc = launch_combine(cv, st, 0xffffffffu, fresh, ChainHints{max_union > 0, 0, slots});
    tap(7);
    return rc;
}

uint64_t b200moe_ffn_workspace_bytes(const b200moe_shape* s, uint32_t capacity) {
    if (!s || check_shape(*s)) return 0;
    return carve_ffn(nullptr, *s, capacity).bytes;
}

int b200moe_ffn(const b200moe_ffn_view* v, void* stream) {
    B200_REQUIRE(v, "null view");
    if (int rc = check_shape(v->shape)) return rc;
    if (int rc = check_policy(v->policy)) return rc;
    const b200moe_shape& s = v->shape;
    B200_REQUIRE(v->policy.experts == s.experts && v->policy.top_k == s.top_k, "ffn: the route policy and the shape disagree on experts / top_k");
    B200_REQUIRE(v->rows <= v->capacity, "ffn: rows %u exceed the workspace capacity %u", v->rows, v->capacity);
    if (v->rows == 0) return B200MOE_OK;
    B200_REQUIRE(v->x && v->y && v->router_weight, "ffn: x / y / router_weight are null");
    B200_REQUIRE(!v->policy.selection_bias || v->select_bias, "ffn: the policy has a selection bias but select_bias is null");
    const FfnScratch F = carve_ffn(v->workspace, s, v->capacity);
    if (!v->workspace || v->workspace_bytes < F.bytes)
        return fail(B200MOE_ERR_WORKSPACE, "ffn: workspace of %llu bytes needed, %llu given", (unsigned long long)F.bytes, (unsigned long long)v->workspace_bytes);
    B200_REQUIRE(aligned(v->workspace, 256), "ffn: workspace must be 256-byte aligned");
    if (!device_ready()) return B200MOE_ERR_CUDA;
    cudaStream_t st = as_stream(stream);

    // The router reads FP32 rows: bfloat16 activations are widened once (exactly) into the workspace (the Qwen prologue's input
    // form, src/cuda/models/qwen/qwen_moe.cu:60-99), by the A8 quantiser where it is a launch of its own, else by a launch before.
    const float* x32 = v->x_is_bf16 ? F.x_f32 : static_cast<const float*>(v->x);
    b200moe_quantize_a8_view q{};
    q.x = x32; q.rows = v->rows; q.width = s.hidden; q.x_stride = s.hidden; q.x_is_bf16 = 0; q.out = F.x;
    b200moe_router_view r{};
    r.x = x32; r.x_stride = s.hidden; r.rows = v->rows; r.hidden = s.hidden;
    r.weight = v->router_weight; r.logit_bias = v->logit_bias; r.bias = v->select_bias; r.policy = v->policy;
    r.logits = F.logits;  // the scores are not asked for
    r.ids = v->ids ? v->ids : F.ids; r.weights = v->route_weights ? v->route_weights : F.weights;
    // Up to 8 rows: one launch for A8 and logits. Up to 32 rows over up to 256 experts: selection and routes share a launch. Over more experts two launches
    // are the faster ones, since a block that both selects and routes has to hold a row's 32 keys a lane beside the routes (512 experts of 2048 x 256, top-8, two
    // launches and one, us a call: 29.2 and 32.8 with 1 row, 46.9 and 54.9 with 8, 81 and 101 with 22).
    const LayerScratch L = carve_layer(F.layer, s, v->capacity);
    const bool fused = select_routes_fusable(r, s.top_k), one_launch = prologue_fusable(r);
    // Where the quantiser is a launch of its own it widens on the way (one pass over the activations instead of two).
    b200moe_quantize_a8_view qb = q;
    qb.x = v->x; qb.x_is_bf16 = 1;
    const bool widen_in_quantizer = v->x_is_bf16 && !one_launch && quantize_a8_vec_ok(qb);
    if (v->x_is_bf16 && !widen_in_quantizer && !one_launch)
        if (int rc = launch_widen_bf16(static_cast<const u16*>(v->x), F.x_f32, u64(v->rows) * s.hidden, st)) return rc;
    b200moe_routes_view rv{};
    if (fused) {
        u32* row_status = v->row_status ? v->row_status : L.row_status;
        rv.ids = r.ids; rv.rows = v->rows; rv.top_k = s.top_k; rv.experts = s.experts;
        rv.split = v->part_experts ? v->part_experts : s.experts / 2;
        rv.scratch = L.routes_scratch; rv.row_status = row_status; rv.out = L.routes;
    }
    if (one_launch) {
        if (int rc = launch_prologue(r, v->x_is_bf16 ? qb : q, st)) return rc;  // widens on the way
    } else {
        if (widen_in_quantizer)
            if (int rc = launch_quantize_a8(qb, st, F.x_f32, s.hidden)) return rc;
        if (int rc = launch_router_logits(r, st, widen_in_quantizer ? nullptr : &q)) return rc;
    }
    if (int rc = fused ? launch_select_routes(r, rv, clear_of(L, v->row_status, v->summary), st) : launch_router_select(r, st)) return rc;

    b200moe_layer_view lv{};
    lv.shape = s; lv.weights = v->weights; lv.rows = v->rows; lv.x = F.x; lv.ids = r.ids; lv.route_weights = r.weights;
    lv.shared = v->shared; lv.combine_form = v->combine_form; lv.parts = v->parts; lv.part_experts = v->part_experts; lv.only_part = -1;
    lv.y = v->y; lv.y_bf16 = v->y_bf16; lv.row_status = v->row_status;
    lv.workspace = F.layer; lv.workspace_bytes = v->workspace_bytes - (static_cast<unsigned char*>(F.layer) - static_cast<unsigned char*>(v->workspace));
    lv.capacity = v->capacity; lv.grouped_min_rows = v->grouped_min_rows; lv.stage_events = v->stage_events;
    lv.summary = v->summary;
    return layer_impl(&lv, stream, fused, false);
}

int b200moe_ffn_host(const b200moe_ffn_view* v, const void* x_host, float* y_host, void* stream) {
    B200_REQUIRE(v && x_host && y_host, "ffn_host: null view / host buffers");
    if (int rc = check_shape(v->shape)) return rc;
    B200_REQUIRE(v->rows <= v->capacity, "ffn_host: rows %u exceed the workspace capacity %u", v->rows, v->capacity);
    const FfnScratch F = carve_ffn(v->workspace, v->shape, v->capacity);
    if (!v->workspace || v->workspace_bytes < F.bytes)
        return fail(B200MOE_ERR_WORKSPACE, "ffn_host: workspace of %llu bytes needed, %llu given", (unsigned long long)F.bytes, (unsigned long long)v->workspace_bytes);
    if (!device_ready()) return B200MOE_ERR_CUDA;
    cudaStream_t st = as_stream(stream);
    const u64 n = u64(v->rows) * v->shape.hidden;
    cudaError_t e = cudaMemcpyAsync(F.x_dev, x_host, n * (v->x_is_bf16 ? 2 : 4), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return fail(B200MOE_ERR_CUDA, "ffn_host: H2D copy: %s", cudaGetErrorString(e));
    b200moe_ffn_view d = *v;
    d.x = F.x_dev; d.y = F.y_dev;
    if (int rc = b200moe_ffn(&d, stream)) return rc;
    e = cudaMemcpyAsync(y_host, F.y_dev, n * 4, cudaMemcpyDeviceToHost, st);
    u32 job = 0;  // the job summary, read back with y: a bounded device wait that ran out must not look like success
    const u32* summary = v->summary ? v->summary : carve_layer(F.layer, v->shape, v->capacity).summary;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&job, summary, sizeof job, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(B200MOE_ERR_CUDA, "ffn_host: D2H copy / synchronize: %s", cudaGetErrorString(e));
    if (job & B200MOE_JOB_WAIT_ABORTED) return fail(B200MOE_ERR_ABORTED, "ffn_host: a bounded device wait ran out (job summary 0x%x); y_host is not valid", job);
    return B200MOE_OK;
}

static int dense_impl(const b200moe_dense_view* v, void* stream, bool fresh);
int b200moe_dense_ffn(const b200moe_dense_view* v, void* stream) { return dense_impl(v, stream, false); }
int b200moe_dense_ffn_fresh(const b200moe_dense_view* v, void* stream) { return dense_impl(v, stream, true); }
static int dense_impl(const b200moe_dense_view* v, void* stream, bool fresh) {
    B200_REQUIRE(v, "null view");
    B200_REQUIRE(v->shape.experts == 1 && v->shape.top_k == 1, "dense_ffn: shape.experts and shape.top_k must be 1");
    if (int rc = check_shape(v->shape)) return rc;
    const b200moe_shape& s = v->shape;
    if (v->rows == 0) return B200MOE_OK;
    B200_REQUIRE(v->y, "dense_ffn: y is null");
    B200_REQUIRE(v->weights.gate && v->weights.up && v->weights.down, "dense_ffn: tensors are null");
    B200_REQUIRE(aligned(v->weights.gate, 16) && aligned(v->weights.up, 16) && aligned(v->weights.down, 16), "dense_ffn: tensors must be 16-byte aligned");
    if (int rc = check_a8(v->x, v->rows, s.hidden, is_kquant(s.gate_type), "dense_ffn x")) return rc;
    const LayerScratch L = carve_layer(v->workspace, s, v->rows);
    if (!v->workspace || v->workspace_bytes < L.bytes)
        return fail(B200MOE_ERR_WORKSPACE, "dense_ffn: workspace of %llu bytes needed, %llu given", (unsigned long long)L.bytes, (unsigned long long)v->workspace_bytes);
    if (!device_ready()) return B200MOE_ERR_CUDA;
    cudaStream_t st = as_stream(stream);
    // every row is one entry of the single expert (slot = row): the routes are written directly, the status words with them; y is zero until down writes it
    if (int rc = launch_dense_routes(L.routes, v->rows, L.row_status, L.summary, fresh ? v->y : nullptr, u64(v->rows) * s.hidden, st)) return rc;
    b200moe_gate_up_view gu{};
    gu.shape = s; gu.weights = v->weights; gu.routes = L.routes; gu.max_union = 1; gu.x = v->x; gu.act = L.act;
    gu.row_status = L.row_status; gu.summary = L.summary;
    if (int rc = enqueue_gate_up(gu, v->rows, st, 0, ChainHints{false, v->rows, v->rows})) return rc;
    b200moe_down_view dn{};
    dn.shape = s; dn.weights = v->weights; dn.routes = L.routes; dn.max_union = 1; dn.act = L.act; dn.raw = v->y; dn.summary = L.summary;
    if (int rc = enqueue_down(dn, v->rows, st, 0, ChainHints{true, v->rows, v->rows})) return rc;
    if (v->y_bf16) {
        // bfloat16 RNE copy of y through the FMA_SLOTS combine with unit weights: fma(1, y, +0) = y exactly
        float* ones = reinterpret_cast<float*>(L.aux);  // the ids are no longer read once the routes exist
        if (int rc = launch_fill_u32(L.aux, 0x3f800000u, v->rows, st)) return rc;
        b200moe_combine_view cv{};
        cv.raw = v->y; cv.weights = ones; cv.rows = v->rows; cv.top_k = 1; cv.hidden = s.hidden; cv.form = B200MOE_COMBINE_FMA_SLOTS;
        cv.only_part = -1; cv.y = L.raw; cv.y_bf16 = v->y_bf16;
        return launch_combine(cv, st);
    }
    return B200MOE_OK;
}

}  // extern "C"

// ---- the launch-record seam (include/strix/weight/resolve.hpp:67-76, src/cuda/weight/registry.hpp:53-65) ----------------
namespace {
using SiteLaunch = int (*)(const void*, void*);
struct SiteRow { b200moe_registration reg; SiteLaunch launch; };
template <class View, int (*Fn)(const View*, void*)>
int site_thunk(const void* view, void* stream) { return Fn(static_cast<const View*>(view), stream); }
#define B200_SITE(id, View, fn) SiteRow{{id, B200MOE_ABI_VERSION, sizeof(View), alignof(View), #fn}, &site_thunk<View, fn>}
const SiteRow kSites[] = {
    B200_SITE(B200MOE_SITE_QUANTIZE_A8, b200moe_quantize_a8_view, b200moe_quantize_a8),
    B200_SITE(B200MOE_SITE_RMSNORM_A8, b200moe_rmsnorm_view, b200moe_rmsnorm_a8),
    B200_SITE(B200MOE_SITE_Q8_0_A8, b200moe_q8a8_view, b200moe_q8_0_a8),
    B200_SITE(B200MOE_SITE_ROUTER, b200moe_router_view, b200moe_router),
    B200_SITE(B200MOE_SITE_ROUTES, b200moe_routes_view, b200moe_build_routes),
    B200_SITE(B200MOE_SITE_ROUTES_STATIC, b200moe_routes_view, b200moe_build_routes_static),
    B200_SITE(B200MOE_SITE_GATE_UP, b200moe_gate_up_view, b200moe_gate_up),
    B200_SITE(B200MOE_SITE_DOWN, b200moe_down_view, b200moe_down),
    B200_SITE(B200MOE_SITE_COMBINE, b200moe_combine_view, b200moe_combine),
    B200_SITE(B200MOE_SITE_LAYER, b200moe_layer_view, b200moe_layer),
    B200_SITE(B200MOE_SITE_FFN, b200moe_ffn_view, b200moe_ffn),
    B200_SITE(B200MOE_SITE_DENSE_FFN, b200moe_dense_view, b200moe_dense_ffn),
};
#undef B200_SITE
constexpr uint32_t kSiteCount = sizeof(kSites) / sizeof(kSites[0]);
}  // namespace

extern "C" {

uint32_t b200moe_registry(const b200moe_registration** rows) {
    static b200moe_registration table[kSiteCount];
    static const bool filled = [] { for (uint32_t i = 0; i < kSiteCount; ++i) table[i] = kSites[i].reg; return true; }();
    (void)filled;
    if (rows) *rows = table;
    return kSiteCount;
}

int b200moe_enqueue(const b200moe_kernel_arguments* a, void* stream) {
    B200_REQUIRE(a, "enqueue: null launch record");
    for (const SiteRow& row : kSites) {
        if (row.reg.schema != a->schema) continue;
        B200_REQUIRE(a->abi_revision == row.reg.revision, "enqueue(%s): launch record of ABI revision %u, this build is revision %u", row.reg.name,
                     a->abi_revision, row.reg.revision);
        B200_REQUIRE(a->bytes == row.reg.bytes, "enqueue(%s): launch record of %llu bytes, the view has %llu", row.reg.name, (unsigned long long)a->bytes,
                     (unsigned long long)row.reg.bytes);
        B200_REQUIRE(a->data && reinterpret_cast<uintptr_t>(a->data) % row.reg.alignment == 0, "enqueue(%s): the view is null or not aligned to %llu bytes",
                     row.reg.name, (unsigned long long)row.reg.alignment);
        return row.launch(a->data, stream);
    }
    return fail(B200MOE_ERR_INVALID_ARGUMENT, "enqueue: unknown schema %u", a->schema);
}

}  // extern "C"

extern "C" {

int b200moe_merge_first_error(b200moe_first_error* record, const uint32_t* summary, uint32_t domain, void* stream) {
    B200_REQUIRE(record && summary, "merge_first_error: record / summary are null");
    B200_REQUIRE(domain == B200MOE_DOMAIN_LEGACY || domain == B200MOE_DOMAIN_Q4K_A8, "merge_first_error: domain %u is not one this library publishes", domain);
    if (!device_ready()) return B200MOE_ERR_CUDA;
    return launch_merge_first_error(record, summary, domain, as_stream(stream));
}

int b200moe_check_first_error(const b200moe_first_error* r) {
    B200_REQUIRE(r, "check_first_error: null record");
    if (r->domain == B200MOE_DOMAIN_NONE && r->bits == 0) return B200MOE_OK;
    if (r->domain == B200MOE_DOMAIN_LEGACY && r->bits != 0)
        return fail(B200MOE_ERR_INVALID_ARGUMENT, "routed experts rejected invalid routes or nonfinite weights (status bits %u)", r->bits);
    if (r->domain == B200MOE_DOMAIN_Q4K_A8 && r->bits != 0)
        return fail(B200MOE_ERR_INVALID_ARGUMENT, "Q4K A8 rejected status bits (route/weight=1,input=2,delta=4,pipeline=8%s): %u",
                    (r->bits & B200MOE_JOB_WAIT_ABORTED) ? ", bounded wait ran out=0x40000000" : "", r->bits);
    return fail(B200MOE_ERR_UNSUPPORTED, "deferred MoE completion record is malformed (domain %u, bits %u)", r->domain, r->bits);
}

}  // extern "C"
