// A residual sum written by its branch's last convolution: every value and gradient of the graph can still be read back.
// Two graphs over the same variables, with gradients shared at the join (the convolution may write the sum) and copied (it
// may not), have to agree to the bit.  Prints "ok" or what differs.
#include <cstdio>
#include <cstring>

#include "arraydiff/op.hh"

using namespace arraydiff;

typedef GPUArray4D<float> Kernel;
typedef GPUArray1D<float> Bias;

struct Graph {
  shared_ptr<CudnnConv2DOpF> trunk, branch;
  ActVar sum, top;   // top: a sum over the sum
};

static size_t failures = 0;
static void same(const char* what, const vector<float>& a, const vector<float>& b, bool equal = true) {
  if ((std::memcmp(a.data(), b.data(), a.size() * 4) == 0) != equal) { std::printf("%s: %s\n", what, equal ? "differs" : "equal"); ++failures; }
}

int main() {
  const size_t W = 21, H = 13, C = 64, N = 2, n = W * H * C * N;
  auto ctx = MultiGPUContext::Make({0}, COMPUTE_BF16_NHWC, (size_t)256 << 20);
  std::mt19937_64 rng(7);
  std::normal_distribution<float> dist(0.f, 1.f);
  auto draw = [&](size_t count, float scale) {
    vector<float> v(count);
    for (auto& x : v) x = dist(rng) * scale;
    return v;
  };
  auto in = IOOp<Act>::Make(Shape3D(W, H, C), N, nullptr, 0, ctx);
  vector<shared_ptr<IOOp<Kernel>>> k;
  for (size_t i = 0; i < 2; ++i) k.push_back(IOOp<Kernel>::Make(Shape4D(1, 1, C, C), 0, nullptr, 0, ctx));
  auto bias = IOOp<Bias>::Make(Shape1D(C), 0, nullptr, 0, ctx);
  Conv2DShape s;
  s.filters = C;
  // what the branch reads, what it is added to, its bias: results of the graph, or variables that a caller loads
  auto make = [&](bool loaded_input, bool loaded_addend, bool with_bias, JoinGrad last) {
    Graph g;
    g.trunk = CudnnConv2DOpF::Make(s, in, k[0], nullptr, ctx);
    g.branch = CudnnConv2DOpF::Make(s, loaded_input ? ActVar(in) : ActVar(g.trunk), k[1], with_bias ? bias : nullptr, ctx);
    g.sum = SumJoinOpF::Make({loaded_addend ? ActVar(in) : ActVar(g.trunk), g.branch}, ctx, {kJoinCopy, last});
    g.top = SumJoinOpF::Make({ActVar(g.trunk), g.sum}, ctx, {kJoinCopy, last});
    return g;
  };
  auto load = [&](shared_ptr<Op> sink, TxnId txn, VarId v, vector<float>& from) {
    VarIdSet set = VarIdSet::Singleton(v);
    any rd = from.data();
    sink->load_val(txn, set, 0, &rd);
  };
  for (int form = 0; form < 8; ++form) {
    const bool loaded_input = form & 1, loaded_addend = form & 2, with_bias = form & 4;
    Graph g[2] = {make(loaded_input, loaded_addend, with_bias, kJoinShare), make(loaded_input, loaded_addend, with_bias, kJoinCopy)};
    auto sink = std::make_shared<GroupSinkOp>(vector<shared_ptr<Op>>{g[0].top, g[1].top});
    auto read = [&](TxnId txn, ActVar v) {
      VarIdSet set = VarIdSet::Singleton(v->data().val.var());
      vector<float> out(n);
      any w = out.data();
      if (sink->store_val(txn, set, 0, &w) != n) { std::printf("form %d: size\n", form); ++failures; }
      return out;
    };
    for (int pass = 0; pass < 2; ++pass) {
      vector<float> x = draw(n, 1.f), b = draw(C, 1.f), w0 = draw(C * C, 0.125f), w1 = draw(C * C, 0.125f);
      TxnId txn;
      load(sink, txn, in->data().val.var(), x);
      load(sink, txn, k[0]->data().val.var(), w0);
      load(sink, txn, k[1]->data().val.var(), w1);
      if (with_bias) load(sink, txn, bias->data().val.var(), b);
      sink->eval(txn);
      const vector<float> sum = read(txn, g[0].sum), conv = read(txn, g[0].branch);
      same("sum", sum, read(txn, g[1].sum));
      same("top", read(txn, g[0].top), read(txn, g[1].top));
      same("convolution", conv, read(txn, g[1].branch));
      same("convolution and sum", conv, sum, false);
      same("sum after the convolution was read", sum, read(txn, g[0].sum));
      {
        // both in one walk: two variables, two extents
        VarIdSet set = VarIdSet::Singleton(g[0].branch->data().val.var());
        set.insert(g[0].sum->data().val.var());
        vector<float> out(2 * n);
        any w = out.data();
        if (sink->store_val(txn, set, 0, &w) != 2 * n) { std::printf("form %d: size of two\n", form); ++failures; }
        same("first of two", vector<float>(out.begin(), out.begin() + n), conv);
        same("second of two", vector<float>(out.begin() + n, out.end()), sum);
      }
      {
        // gradients: of the top (loaded), the sum and the branch's output (the same)
        vector<float> dy = draw(n, 1.f);
        VarIdSet sums = VarIdSet::Singleton(g[0].top->data().grad.var());
        sums.insert(g[1].top->data().grad.var());
        vector<float> both(dy);
        both.insert(both.end(), dy.begin(), dy.end());
        any rd = both.data();
        sink->load_grad(txn, sums, 0, &rd);
        sink->backward(txn);
        vector<float> of[2];
        for (int i = 0; i < 2; ++i) {
          VarIdSet set = VarIdSet::Singleton(g[i].branch->data().grad.var());
          set.insert(g[i].sum->data().grad.var());
          set.insert(g[i].trunk->data().grad.var());
          of[i].resize(3 * n);
          any w = of[i].data();
          if (sink->store_grad(txn, set, 0, &w) != 3 * n) { std::printf("form %d: size of three gradients\n", form); ++failures; }
        }
        same("gradients of trunk, branch and sum", of[0], of[1]);
      }
      // the next batch and other parameters are loaded, nothing is evaluated: results are those of the last pass
      vector<float> x2 = draw(n, 1.f), b2 = draw(C, 1.f), v0 = draw(C * C, 0.125f), v1 = draw(C * C, 0.125f);
      TxnId next;
      load(sink, next, in->data().val.var(), x2);
      load(sink, next, k[0]->data().val.var(), v0);
      load(sink, next, k[1]->data().val.var(), v1);
      if (with_bias) load(sink, next, bias->data().val.var(), b2);
      same("convolution before the next pass", conv, read(next, g[0].branch));
      same("sum before the next pass", sum, read(next, g[0].sum));
    }
  }
  const int status = ctx->device_context(0)->read_status();
  if (status) { std::printf("status %d\n", status); ++failures; }
  if (!failures) std::printf("ok\n");
  return failures ? 1 : 0;
}
