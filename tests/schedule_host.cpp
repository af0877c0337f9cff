// Host side of the scheduled runs without a GPU (test helper, built by test_schedule_host.py): the runtime's own source
// with the CUDA runtime replaced by host memory, so that contexts, their offset tables and the launches of their run
// ranges are the real ones.  Reads lines from stdin and answers each with a line that starts with "ok" or "bad".
//
//   sched METHOD froz occ_a occ_b orbs rhf act_occ_b act_unocc_a deep
//     every range's schedule: dependencies name earlier launches; the items of a shared launch cover their
//     contractions' products once; in one shared launch an element is stored once or only added to.  deep: for every
//     element, two launches of which one stores, or one reads and one writes, are ordered by the dependencies.
//   copies
//     two threads read two large pageable blocks of one context at the same time.
#include "../ccq_b200/csrc/runtime.cu"

#include <sys/mman.h>
#include <unistd.h>

#include <iostream>
#include <set>
#include <unordered_map>
#include <unordered_set>

// ---- the CUDA runtime on host memory: streams run at once, launches do nothing -----------------------------
namespace {
bool slow = false;   // a transfer takes time
std::mutex mem_mutex;
std::map<void *, size_t> mem;
cudaError_t get(void **p, size_t n) {
    *p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (*p == MAP_FAILED) return cudaErrorMemoryAllocation;
    std::lock_guard<std::mutex> l(mem_mutex);
    mem[*p] = n;
    return cudaSuccess;
}
cudaError_t put(void *p) {
    std::lock_guard<std::mutex> l(mem_mutex);
    if (!mem.count(p)) return cudaSuccess;
    munmap(p, mem[p]);
    mem.erase(p);
    return cudaSuccess;
}
template <typename T>
cudaError_t handle(T *h) {
    static int x;
    *h = reinterpret_cast<T>(&x);
    return cudaSuccess;
}
}  // namespace

extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 0; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    if (slow) usleep(100);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return get(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return get(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return get(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return get(p, n); }
cudaError_t cudaFree(void *p) { return put(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return put(p); }
cudaError_t cudaFreeHost(void *p) { return put(p); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }   // memory starts at zero
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **, unsigned long long, cudaDriverEntryPointQueryResult *) {
    return cudaErrorNotSupported;
}
}

namespace {

struct Fail : std::runtime_error {
    using std::runtime_error::runtime_error;
};

// one launch's accesses to elements; items of a shared launch run in any order
struct Access {
    std::vector<const double *> read, add, store;
};

Access item_access(const MultiItem &it, bool reads) {
    Access a;
    if (it.flags >> MI_SHAPE == MS_COPY) {
        for (int i = 0; i < it.m; ++i) {
            a.store.push_back(it.C + i);
            if (reads && it.A) a.read.push_back(it.A + i);
        }
        return a;
    }
    auto &out = it.flags & MI_ADD ? a.add : a.store;
    for (int i = 0; i < it.m; ++i)
        for (int j = 0; j < it.n; ++j) out.push_back(it.C + it.cm[i] + it.cn[j]);
    if (!reads) return a;
    for (int k = 0; k < it.k; ++k) {
        for (int i = 0; i < it.m; ++i) a.read.push_back(it.A + it.am[i] + it.ak[k]);
        for (int j = 0; j < it.n; ++j) a.read.push_back(it.B + it.bn[j] + it.bk[k]);
    }
    return a;
}

Access op_access(ccq_b200_ctx *c, const Op &o) {
    Access a;
    auto whole = [&](std::vector<const double *> &v, const std::string &b) {
        const DevBuf &d = c->bufs.at(b);
        for (long long x = 0; x < d.numel; ++x) v.push_back(d.ptr + x);
    };
    auto view = [&](const ViewSpec &v) {
        const Resolved r = resolve(c, v);
        std::vector<const double *> p{r.base};
        for (auto &l : r.order) {
            std::vector<const double *> q;
            for (auto *b : p)
                for (long long x = 0; x < r.extent.at(l); ++x) q.push_back(b + x * r.stride.at(l));
            p.swap(q);
        }
        a.read.insert(a.read.end(), p.begin(), p.end());
    };
    switch (o.kind) {
        case OP_GETT: {
            const GettArgs &g = o.g;
            auto &out = g.beta ? a.add : a.store;
            for (int i = 0; i < g.M; ++i)
                for (int j = 0; j < g.N; ++j) out.push_back(g.C + g.offC_m[i] + g.offC_n[j]);
            std::vector<GettSeg> segs = o.hsegs;
            if (segs.empty()) segs.push_back(GettSeg{g.A, g.B, g.offA_m, g.offA_k, g.offB_n, g.offB_k, g.K, g.alpha});
            for (auto &s : segs)
                for (int k = 0; k < s.K; ++k) {
                    for (int i = 0; i < g.M; ++i) a.read.push_back(s.A + s.offA_m[i] + s.offA_k[k]);
                    for (int j = 0; j < g.N; ++j) a.read.push_back(s.B + s.offB_n[j] + s.offB_k[k]);
                }
            break;
        }
        case OP_ASM:
            if (!o.asmargs.total) break;   // no canonical element
            for (auto &t : o.terms) view(t.second);
            if (o.asmargs.mode != 1) whole(a.read, o.block);
            if (o.asmargs.mode == 2) {
                for (const char *b : {"HDA", "HDB", "ECOR"}) whole(a.read, b);
                whole(a.add, "LN");
            }
            whole(a.store, o.block);
            break;
        case OP_COPY:
            whole(a.read, o.arg1);
            if (o.dress)
                for (int k : {1, 2}) whole(a.read, std::string("T1") + o.arg0[k]);
            whole(a.store, o.arg0);
            break;
        case OP_ZERO:
            whole(a.store, o.arg0);
            break;
        case OP_LENERGY:
            for (const char *b : {"LN", "ECOR"}) whole(a.read, b);
            whole(a.store, "EL");
            break;
        case OP_CRCC:
            for (const char *b : {"M3", "L3"}) whole(a.read, b + o.arg0);
            for (const char *b : {"HDA", "HDB", "H2AA", "H2AB", "H2BB"}) whole(a.read, b);
            whole(a.add, "E23");
            break;
        default: break;
    }
    return a;
}

std::string check(ccq_b200_ctx *c, size_t from, size_t to, bool deep) {
    const Sched s = build_sched(c, from, to);
    const size_t nn = s.nodes.size();
    // dependencies and everything reached through them
    std::vector<std::vector<char>> anc(nn, std::vector<char>(nn, 0));
    for (size_t k = 0; k < nn; ++k)
        for (int d : s.nodes[k].deps) {
            if (d < 0 || d >= (int)k) throw Fail("a dependency is not an earlier launch");
            anc[k][d] = 1;
            for (size_t q = 0; q < (size_t)d; ++q) anc[k][q] |= anc[d][q];
        }
    // products: each contraction in its own launch or in items
    std::set<size_t> own;
    size_t nitems = 0, nstores = 0;
    double items = 0, ops = 0;
    for (auto &n : s.nodes) {
        if (n.kind == SchedNode::OP) {
            own.insert(n.op);
            own.insert(c->plan.ops[n.op].group_ops.begin(), c->plan.ops[n.op].group_ops.end());
        }
        nitems += n.nitems;
        for (size_t q = n.item0; q < n.item0 + n.nitems; ++q) {
            const MultiItem &it = s.items[q];
            if (it.flags >> MI_SHAPE == MS_COPY) continue;
            items += (double)it.m * it.n * it.k;
            nstores += !(it.flags & MI_ADD);
            if (it.k < 1 || it.k > MULTI_K) throw Fail("K range of an item");
        }
    }
    for (size_t i = from; i < to; ++i) {
        const Op &o = c->plan.ops[i];
        if (o.kind == OP_GETT && !o.frozen && !o.dressed && !own.count(i)) ops += (double)o.g.M * o.g.N * o.g.K;
    }
    if (items != ops) throw Fail("products of the items: " + std::to_string(items) + " of " + std::to_string(ops));
    // stores of one shared launch
    for (auto &n : s.nodes) {
        std::unordered_set<const double *> stored;
        for (size_t q = n.item0; q < n.item0 + n.nitems; ++q)
            if (!(s.items[q].flags & MI_ADD))
                for (auto *p : item_access(s.items[q], false).store)
                    if (!stored.insert(p).second) throw Fail("two items of a launch store the same element");
        if (stored.empty()) continue;
        for (size_t q = n.item0; q < n.item0 + n.nitems; ++q)
            for (auto *p : item_access(s.items[q], false).add)
                if (stored.count(p)) throw Fail("an element is stored and added to in one launch");
    }
    if (deep) {
        struct Last {
            int store = -1;
            std::vector<int> add, read;
        };
        std::unordered_map<const double *, Last> last;
        int barrier = -1;
        for (int k = 0; k < (int)nn; ++k) {
            const SchedNode &n = s.nodes[k];
            if (barrier >= 0 && !anc[k][barrier]) throw Fail("a launch does not wait for a barrier");
            std::vector<Access> acc;
            if (n.kind == SchedNode::CLEAR) {
                acc.resize(1);
                const auto &z = c->zero_mem.at(from);
                for (long long x = 0; x < z.second; ++x) acc[0].store.push_back(z.first + x);
            } else if (n.kind == SchedNode::OP) {
                const Op &o = c->plan.ops[n.op];
                if (op_io(c, o, true).barrier) {
                    for (int q = 0; q < k; ++q)   // (it touches no accumulation buffer)
                        if (!anc[k][q] && s.nodes[q].kind != SchedNode::CLEAR) throw Fail("a barrier does not wait for an earlier launch");
                    barrier = k;
                }
                acc.push_back(op_access(c, o));
            } else {
                for (size_t q = n.item0; q < n.item0 + n.nitems; ++q) acc.push_back(item_access(s.items[q], true));
            }
            // k itself counts as unordered, except inside one operation
            auto after = [&](int q) { return q < 0 || (q == k ? n.kind != SchedNode::MULTI : anc[k][q]); };
            auto all_after = [&](const std::vector<int> &v) {
                for (int q : v)
                    if (!after(q)) return false;
                return true;
            };
            auto note = [&](std::vector<int> &v) {
                if (v.empty() || v.back() != k) v.push_back(k);
            };
            const std::string at = " (launch " + std::to_string(k) + " of " + std::to_string(nn) + ")";
            for (auto &a : acc)
                for (auto *p : a.read) {
                    Last &l = last[p];
                    if (!after(l.store) || !all_after(l.add)) throw Fail("read without waiting for a writer" + at);
                    note(l.read);
                }
            for (auto &a : acc)
                for (auto *p : a.add) {
                    Last &l = last[p];
                    if (!after(l.store) || !all_after(l.read)) throw Fail("addition not ordered" + at);
                    note(l.add);
                }
            for (auto &a : acc)
                for (auto *p : a.store) {
                    Last &l = last[p];
                    if (!after(l.store) || !all_after(l.add) || !all_after(l.read)) throw Fail("store not ordered" + at);
                    l.store = k;
                    l.add.clear();
                    l.read.clear();
                }
        }
    }
    return " " + std::to_string(nn) + "/" + std::to_string(nitems) + "/" + std::to_string(nstores);
}

struct Context {
    ccq_b200_ctx *c = nullptr;
    Context(const std::string &method, long long froz, long long oa, long long ob, long long orbs, bool rhf, long long ao,
            long long av) {
        const size_t n = orbs - froz;
        std::vector<double> f(orbs * orbs, 0.0);
        double *v;
        get((void **)&v, 8 * n * n * n * n);
        const ccq_b200_dims d{froz, oa, ob, orbs};
        ccq_b200_init_opts opt{};
        opt.rowmajor = 1;
        opt.act_occ_b = ao;
        opt.act_unocc_a = av;
        const int rc = ccq_b200_init_ex(&d, method.c_str(), &opt, f.data(), f.data(), v, v, v, rhf, 0.0, 5, &c);
        put(v);
        if (rc) throw Fail("init: " + g_last_error);
    }
    ~Context() { ccq_b200_free(c); }
};

std::string copies() {
    Context x("CCSDT", 0, 5, 5, 22, false, -1, -1);
    const char *name[2] = {"T3A", "T3B"};
    const long long n = x.c->bufs.at("T3A").numel;
    if (8 * n < (long long)kCopyMin) throw Fail("blocks too small");
    std::vector<double> put[2], back[2];
    for (int b = 0; b < 2; ++b) {
        put[b].resize(n);
        back[b].resize(n);
        for (long long i = 0; i < n; ++i) put[b][i] = (double)(2 * i + b);
        if (ccq_b200_block(x.c, name[b], put[b].data(), n, 1)) throw Fail(g_last_error);
    }
    slow = true;
    for (int rep = 0; rep < 20; ++rep) {
        std::thread th[2];
        for (int b = 0; b < 2; ++b) {
            std::fill(back[b].begin(), back[b].end(), -1.0);
            th[b] = std::thread([&, b] { ccq_b200_block(x.c, name[b], back[b].data(), n, 0); });
        }
        for (auto &t : th) t.join();
        for (int b = 0; b < 2; ++b)
            if (back[b] != put[b]) throw Fail("a thread read the other's data");
    }
    slow = false;
    return "";
}

}  // namespace

int main() {
    std::string line;
    while (std::getline(std::cin, line)) {
        try {
            std::stringstream ss(line);
            std::string cmd, method, out;
            long long froz, oa, ob, orbs, rhf, ao, av, deep;
            ss >> cmd;
            if (cmd == "copies") {
                out = copies();
            } else {
                ss >> method >> froz >> oa >> ob >> orbs >> rhf >> ao >> av >> deep;
                Context x(method, froz, oa, ob, orbs, rhf != 0, ao, av);
                const auto r = run_ranges(x.c);
                for (size_t k = 0; k + 1 < r.size(); ++k) out += check(x.c, r[k], r[k + 1], deep != 0);
            }
            std::cout << "ok" << out << std::endl;
        } catch (const std::exception &e) {
            std::cout << "bad " << e.what() << std::endl;
        }
    }
}
