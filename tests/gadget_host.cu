// abi_mlwe.cu on a fake engine, for its host-side decisions: which route a gadget product
// takes and what an entry point does when a launch or its scratch fails.  Run without a
// device: no kernel of it may start.
//
//   gadget_host <entry> <case>     prints the engine calls the entry point made
#include <cuda_runtime.h>

// kernel launches report what the case asks for (without a device none of them starts)
static cudaError_t fake_last_error();
#define cudaGetLastError fake_last_error
#include "../vfhe_b200/csrc/abi_mlwe.cu"
#undef cudaGetLastError

#include <stdio.h>
#include <stdlib.h>

#include <map>
#include <utility>
#include <string>

namespace {
std::string g_case;
std::map<std::string, int> g_calls;
void call(const char* name) { ++g_calls[name]; }
}  // namespace

static cudaError_t fake_last_error() { return g_case == "launch_fails" ? cudaErrorInvalidValue : cudaSuccess; }

namespace vc {
Context& ctx() {
    static Context c;
    return c;
}
bool ensure_ready() { return true; }
cudaStream_t stream() { return nullptr; }
bool sync(const char*) { return true; }
void set_error(const char*, const char*) { call("error"); }
bool check_cuda(int code, const char* where) {
    if (code) set_error(where, "");
    return code == 0;
}
void note_launch(int) {}
void* device_alloc(size_t bytes) {
    if (g_case == "no_scratch") {
        call("error");
        return nullptr;
    }
    call("alloc");
    return malloc(bytes);
}
void device_free(void* p) {
    if (p) call("free");
    free(p);
}
void prefetch_to_device(const void*, size_t) {}
int launch_ntt(const RowSet& rows, const PrimeInfo*, bool, cudaStream_t) {
    call(rows.digits ? "digits" : "transform");
    return g_case == "transform_fails" && rows.digits ? (int)cudaErrorInvalidValue : 0;
}
bool ntt_f64_eligible(const RowSet&) { return true; }
int launch_ew(EwOp, const EwSet&, const PrimeInfo*, cudaStream_t) {
    call("zero");
    return 0;
}
void op_product(Poly*, Poly*, Poly*, int, const char*) { call("product"); }
void op_round_divide(Poly* const*, int, uint64_t, const char*) { call("divide"); }
Poly* poly_create(uint64_t, uint64_t mask, IncNtt* t) {
    Poly* p = new Poly();
    p->base = (uint64_t*)calloc(t->pub.l * t->pub.N, 8);
    p->pub.coeffs = (uint64_t**)malloc(sizeof(uint64_t*) * t->pub.l);
    for (uint64_t i = 0; i < t->pub.l; ++i) p->pub.coeffs[i] = p->base + i * t->pub.N;
    p->pub.ntt = &t->pub;
    p->pub.rns_mask = mask;
    p->pub.allocated_l = t->pub.l;
    return p;
}
void poly_destroy(Poly* p) {
    free(p->base);
    free(p->pub.coeffs);
    delete p;
}
}  // namespace vc

extern "C" {
void polynomial_RNSc_mod_reduce_lifted(void*, void*, uint64_t) {}
void polynomial_RNSc_to_RNS(void*, void*) {}
void polynomial_RNS_to_RNSc(void*, void*) {}
void polynomial_add_RNSc_polynomial(void*, void*, void*) { call("add"); }
}

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    int devices = 0;
    if (cudaGetDeviceCount(&devices) == cudaSuccess && devices > 0) return 3;
    cudaGetLastError();
    const std::string entry = argv[1];
    g_case = argv[2];
    IncNtt t;
    t.pub.N = t.P = 256;
    t.pub.split_degree = 1;
    t.pub.l = 4;
    t.logP = 8;
    t.info.resize(4);
    for (auto& p : t.info) p.fp64 = 1;
    const uint64_t ct = 0b0111, ext = 0b1111;  // limbs 0..2, the special prime at 3
    RNS_MLWE in = new_mlwe(256, 1, ct, &t), out = new_mlwe(256, 1, ct, &t), key[6];
    for (auto& k : key) k = new_mlwe(256, 1, ext, &t);
    if (g_case == "large_digit") {  // a digit of a prime above 2^50 that the keys do not carry
        t.info[1].fp64 = 0;
        for (auto& k : key) k->a[0]->rns_mask = k->b->rns_mask = 0b1101;
    }
    // operands that share a polynomial
    if (g_case == "key_mask_is_output_body") key[1]->a[0] = out->b;
    if (g_case == "key_body_is_output_mask") key[2]->b = out->a[0];
    if (g_case == "output_mask_is_output_body") out->a[0] = out->b;
    if (g_case == "input_body_is_output_mask") in->b = out->a[0];
    if (g_case == "input_body_is_output_body") in->b = out->b;
    if (g_case == "input_mask_is_output_body") in->a[0] = out->b;
    // rows that do not lie one after the other in the polynomial's block
    auto swap_rows = [](RNS_Polynomial p) { std::swap(p->coeffs[0], p->coeffs[2]); };
    if (g_case == "key_rows_moved") swap_rows(key[1]->b);
    if (g_case == "output_rows_moved") swap_rows(out->a[0]);
    if (g_case == "digit_rows_moved") swap_rows(in->a[0]);
    if (entry == "keyswitch") {
        void* comp[1] = {key};
        mlwe_RNSc_GHS_hybrid_keyswitch(out, in, comp, 0);
    } else {
        mgsw_external_product(out, key, in, 3, 1);
    }
    for (auto& c : g_calls) printf("%s %d\n", c.first.c_str(), c.second);
    return 0;
}
