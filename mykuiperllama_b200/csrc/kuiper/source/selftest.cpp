// Built-in checks of the base / tensor / op classes, reachable through kuiper_selftest().
//
// They restate, against this implementation, what the reference's unit tests pin:
// buffers (test/test_tensor/test_buffer.cpp:7-114: ownership flags, allocator identity,
// device tags, copy_from in the three CUDA directions), tensors
// (test/test_tensor/test_tensor.cpp:6-276: constructors of every rank, strides, clone,
// to_cpu / to_cuda, borrowed pointers, assgin) and the add operator through the kernel
// registry (test/test_op/test_op_add.cpp:7-91) plus the VecAddLayer the reference never
// exercises.  gtest is not a dependency here: each EXPECT appends a line to the report.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <sstream>
#include <vector>

#include "kuiper_llama.h"
#include "op/add.h"
#include "op/kernel/kernel_interface.h"
#include "op/matmul.h"
#include "tensor/tensor.h"

namespace {

struct Report {
    std::ostringstream out;
    int failed = 0;
    int passed = 0;
    void expect(bool ok, const char* expr, const char* file, int line) {
        if (ok) {
            passed++;
        } else {
            failed++;
            out << "FAILED " << file << ":" << line << " " << expr << "\n";
        }
    }
};

#define EXPECT(cond) rep.expect((cond), #cond, __FILE__, __LINE__)

using base::DataType;
using base::DeviceType;
using tensor::Tensor;

void fill_device(float* dev, size_t n, float v) {
    std::vector<float> h(n, v);
    cudaMemcpy(dev, h.data(), n * sizeof(float), cudaMemcpyHostToDevice);
}

bool all_equal_device(const float* dev, size_t n, float v, float tol = 0.f) {
    std::vector<float> h(n);
    cudaMemcpy(h.data(), dev, n * sizeof(float), cudaMemcpyDeviceToHost);
    for (float x : h)
        if (!(x >= v - tol && x <= v + tol)) return false;
    return true;
}

void test_status(Report& rep) {
    base::Status ok = base::error::success();
    base::Status bad = base::error::invalid_argument("nope");
    EXPECT(bool(ok) && int(ok) == 0);
    EXPECT(!bool(bad) && bad == base::StatusCode::InvalidArgument && bad.get_err_msg() == "nope");
    EXPECT(base::error::key_has_exits().get_err_code() == 6 && base::error::internal_error().get_err_code() == 5);
    EXPECT(base::data_type_size(DataType::DataTypeFp32) == 4 && base::data_type_size(DataType::DataTypeInt8) == 1 &&
           base::data_type_size(DataType::DataTypeInt32) == 4 && base::data_type_size(DataType::DataTypeBf16) == 2 &&
           base::data_type_size(DataType::DataTypeFp16) == 2);
}

void test_buffer_cpu(Report& rep) {
    auto alloc = base::CPUDeviceAllocatorFactory::get_instance();
    base::Buffer buffer(32, alloc);
    EXPECT(buffer.ptr() != nullptr && buffer.byte_size() == 32 && !buffer.is_external());
    EXPECT(buffer.allocator() == alloc && buffer.device_type() == DeviceType::DeviceCPU);
    buffer.set_device_type(DeviceType::DeviceCUDA);
    EXPECT(buffer.device_type() == DeviceType::DeviceCUDA);

    float* raw = new float[32];
    {
        base::Buffer ext(32, nullptr, raw, true);
        EXPECT(ext.is_external() && ext.byte_size() == 32 && ext.ptr() == raw);
    }
    raw[0] = 1.f;  // still ours: a borrowed buffer never frees
    delete[] raw;

    auto shared = std::make_shared<base::Buffer>(16, alloc);
    EXPECT(shared->get_shared_from_this() == shared);
}

void test_tensor_cpu(Report& rep) {
    auto alloc = base::CPUDeviceAllocatorFactory::get_instance();
    Tensor t3(DataType::DataTypeFp32, 32, 32, 3, true, alloc);
    EXPECT(!t3.is_empty() && t3.dims_size() == 3 && t3.size() == 32u * 32 * 3);
    EXPECT(t3.strides() == std::vector<size_t>({96, 3, 1}));
    EXPECT(t3.byte_size() == t3.size() * 4 && t3.device_type() == DeviceType::DeviceCPU);

    Tensor t5(DataType::DataTypeFp32, std::vector<int32_t>{2, 3, 4, 5, 6}, true, alloc);
    EXPECT(t5.dims_size() == 5 && t5.size() == 720 && t5.strides() == std::vector<size_t>({360, 120, 30, 6, 1}));

    // borrowed pointer: device tag is set by hand, pointer arithmetic in elements
    float* raw = new float[32];
    raw[0] = 31;
    raw[1] = 32;
    Tensor tb(DataType::DataTypeFp32, 32, false, nullptr, raw);
    EXPECT(tb.device_type() == DeviceType::DeviceUnknown);
    tb.set_device_type(DeviceType::DeviceCPU);
    EXPECT(tb.device_type() == DeviceType::DeviceCPU && tb.ptr<float>() == raw && *tb.ptr<float>(1) == 32);
    EXPECT(tb.get_buffer()->is_external());

    // clone is deep
    Tensor t1(DataType::DataTypeFp32, 32, 32, true, alloc);
    for (size_t i = 0; i < t1.size(); i++) t1.index<float>(int64_t(i)) = 1.f;
    Tensor t2 = t1.clone();
    t2.index<float>(0) = 7.f;
    EXPECT(t1.index<float>(0) == 1.f && t2.index<float>(1) == 1.f && t2.ptr<float>() != t1.ptr<float>());
    EXPECT(t2.dims() == t1.dims() && t2.data_type() == t1.data_type() && t2.byte_size() == t1.byte_size());

    // assgin accepts a buffer that is large enough, refuses one that is too small
    auto big = std::make_shared<base::Buffer>(32 * 32 * 4, nullptr, new float[32 * 32], true);
    big->set_device_type(DeviceType::DeviceCPU);
    EXPECT(t1.assgin(big) && t1.ptr<void>() == big->ptr() && t1.size() == 32u * 32);
    auto small = std::make_shared<base::Buffer>(16, alloc);
    EXPECT(!t1.assgin(small));
    delete[] static_cast<float*>(big->ptr());

    // reshape grows by copy and keeps contents
    Tensor tr(DataType::DataTypeFp32, 4, true, alloc);
    for (int i = 0; i < 4; i++) tr.index<float>(i) = float(i);
    tr.reshape({2, 4});
    EXPECT(tr.size() == 8 && tr.index<float>(3) == 3.f && tr.dims() == std::vector<int32_t>({2, 4}));
    tr.reset(DataType::DataTypeInt32, {3});
    EXPECT(tr.is_empty() && tr.size() == 3 && tr.data_type() == DataType::DataTypeInt32);
    delete[] raw;
}

void test_layer_cpu(Report& rep) {
    // slot bookkeeping and argument checking need no device
    op::MatmulLayer mm(DeviceType::DeviceCUDA, 256, 128, true);
    EXPECT(mm.weights_size() == 2 && mm.input_size() == 1 && mm.output_size() == 1 && mm.group_size() == 128);
    EXPECT(mm.layer_type() == op::LayerType::LayerMatmul && mm.data_type() == DataType::DataTypeFp32);
    mm.set_residual(true);
    EXPECT(mm.input_size() == 2);
    base::Status st = mm.check();  // nothing bound yet
    EXPECT(!st && st == base::StatusCode::InvalidArgument);
    auto alloc = base::CPUDeviceAllocatorFactory::get_instance();
    Tensor wrong(DataType::DataTypeFp32, 4, true, alloc);
    EXPECT(!mm.set_weight(0, wrong));  // fp32 is not the packed INT4 word type
    op::VecAddLayer add(DeviceType::DeviceCUDA);
    EXPECT(add.input_size() == 2 && add.output_size() == 1 && add.layer_name() == "Add");
    EXPECT(!add.forward());  // empty tensors are rejected by check()
}

void test_cuda(Report& rep) {
    auto cu = base::CUDADeviceAllocatorFactory::get_instance();
    auto cpu = base::CPUDeviceAllocatorFactory::get_instance();
    {
        base::Buffer b(32, cu);
        EXPECT(b.ptr() != nullptr && !b.is_external() && b.device_type() == DeviceType::DeviceCUDA && b.allocator() == cu);
    }
    {  // copy_from: host -> device -> device -> host
        const int n = 32;
        base::Buffer host(n * 4, cpu), d1(n * 4, cu), d2(n * 4, cu), back(n * 4, cpu);
        float* hp = static_cast<float*>(host.ptr());
        for (int i = 0; i < n; i++) hp[i] = float(i);
        d1.copy_from(host);
        d2.copy_from(&d1);
        back.copy_from(d2);
        bool same = true;
        for (int i = 0; i < n; i++) same = same && static_cast<float*>(back.ptr())[i] == float(i);
        EXPECT(same);
    }
    {  // to_cpu / to_cuda / clone on the device
        Tensor t(DataType::DataTypeFp32, 32, 32, true, cu);
        fill_device(t.ptr<float>(), t.size(), 1.f);
        Tensor c = t.clone();
        EXPECT(c.device_type() == DeviceType::DeviceCUDA && c.ptr<float>() != t.ptr<float>() &&
               all_equal_device(c.ptr<float>(), c.size(), 1.f));
        t.to_cpu();
        EXPECT(t.device_type() == DeviceType::DeviceCPU && t.index<float>(1023) == 1.f);
        t.to_cuda();
        EXPECT(t.device_type() == DeviceType::DeviceCUDA && all_equal_device(t.ptr<float>(), t.size(), 1.f));
    }
    {  // arena: no driver call per allocation, 256-byte granularity, exhaustion is reported by CHECK
        auto arena = std::make_shared<base::CUDAArenaAllocator>(4096);
        Tensor a(DataType::DataTypeFp32, 10, true, arena), b(DataType::DataTypeFp32, 10, true, arena);
        EXPECT(a.ptr<char>() + 256 == b.ptr<char>() && arena->used() == 512);
    }
    // add through the registry, default stream and user stream, plus the unaligned tail case
    for (int variant = 0; variant < 3; variant++) {
        const bool big = variant == 2;
        Tensor a = big ? Tensor(DataType::DataTypeFp32, 32, 151, 13, true, cu) : Tensor(DataType::DataTypeFp32, 32, 151, true, cu);
        Tensor b = a.clone(), out = a.clone();
        fill_device(a.ptr<float>(), a.size(), big ? 2.1f : 2.f);
        fill_device(b.ptr<float>(), b.size(), big ? 3.3f : 3.f);
        cudaStream_t s = nullptr;
        if (variant == 1) cudaStreamCreate(&s);
        kernel::get_add_kernel(DeviceType::DeviceCUDA)(a, b, out, s);
        cudaDeviceSynchronize();
        EXPECT(all_equal_device(out.ptr<float>(), out.size(), big ? 5.4f : 5.f, big ? 1e-4f : 0.f));
        if (s) cudaStreamDestroy(s);
    }
    {  // the layer path the reference never tests
        op::VecAddLayer add(DeviceType::DeviceCUDA);
        auto cfg = std::make_shared<kernel::CudaConfig>();
        cfg->create();
        add.set_cuda_config(cfg);
        Tensor a(DataType::DataTypeFp32, 1000, true, cu), b(DataType::DataTypeFp32, 1000, true, cu),
            out(DataType::DataTypeFp32, 1000, true, cu);
        fill_device(a.ptr<float>(), 1000, 2.f);
        fill_device(b.ptr<float>(), 1000, 3.f);
        EXPECT(bool(add.forward(a, b, out)));
        cudaStreamSynchronize(cfg->stream());
        EXPECT(all_equal_device(out.ptr<float>(), 1000, 5.f));
        Tensor short_out(DataType::DataTypeFp32, 999, true, cu);
        EXPECT(!add.forward(a, b, short_out));
    }
}

// a quantised projection with its operands on both sides: random packed words, scales of about 2^-7, inputs in [-1, 1)
struct QuantCase {
    int32_t M, K, N;
    std::vector<uint32_t> qw, qz;
    std::vector<uint16_t> scales;
    std::vector<float> x;
    Tensor tx, ty;
    op::MatmulLayer layer;
    std::shared_ptr<kernel::CudaConfig> cfg = std::make_shared<kernel::CudaConfig>();

    template <typename T>
    static Tensor upload(DataType type, std::vector<int32_t> dims, const std::vector<T>& v) {
        Tensor t(type, std::move(dims), true, base::CUDADeviceAllocatorFactory::get_instance());
        cudaMemcpy(t.ptr<void>(), v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
        return t;
    }
    QuantCase(Report& rep, int32_t m, int32_t k, int32_t n)
        : M(m), K(k), N(n), qw(size_t(k) * n / 8), qz(size_t(k) / 128 * n / 8), scales(size_t(k) / 128 * n), x(size_t(m) * k),
          layer(DeviceType::DeviceCUDA, n, k, true) {
        uint32_t state = 12345u + uint32_t(m * 7 + k + n);
        auto next = [&] { return (state = state * 1664525u + 1013904223u) >> 8; };  // 24 random bits
        for (uint32_t& w : qw) w = next() ^ (next() << 16);
        for (uint32_t& w : qz) w = next() ^ (next() << 16);
        for (uint16_t& s : scales) s = uint16_t((8u << 10) | (next() & 1023u));
        for (float& v : x) v = float(next()) / 8388608.f - 1.f;
        cfg->create();
        layer.set_cuda_config(cfg);
        EXPECT(bool(layer.set_weight(0, upload(DataType::DataTypeInt32, {K, N / 8}, qw))));
        EXPECT(bool(layer.set_weight(1, upload(DataType::DataTypeInt32, {K / 128, N / 8}, qz))));
        layer.set_scales(upload(DataType::DataTypeFp16, {K / 128, N}, scales));
        layer.set_workspace(scratch(kernel::matmul_quant_workspace_bytes(M, K, N)));
        tx = upload(DataType::DataTypeFp32, {M, K}, x);
        ty = Tensor(DataType::DataTypeFp32, std::vector<int32_t>{M, N}, true, base::CUDADeviceAllocatorFactory::get_instance());
    }
    static Tensor scratch(size_t bytes) {
        Tensor t(DataType::DataTypeFp32, int32_t(bytes / 4 + 1), true, base::CUDADeviceAllocatorFactory::get_instance());
        cudaMemset(t.ptr<void>(), 0, t.byte_size());
        return t;
    }
    std::vector<float> run(Report& rep) {
        cudaMemset(ty.ptr<void>(), 0, ty.byte_size());
        cudaDeviceSynchronize();
        EXPECT(bool(layer.forward(tx, ty)));
        cudaStreamSynchronize(cfg->stream());
        std::vector<float> y(ty.size());
        cudaMemcpy(y.data(), ty.ptr<void>(), ty.byte_size(), cudaMemcpyDeviceToHost);
        return y;
    }
    // largest |y - x . W| over the largest |x . W|, in 64 bits
    double error(const std::vector<float>& y) const {
        static const int place[8] = {0, 4, 1, 5, 2, 6, 3, 7};  // nibble of logical column c
        double worst = 0, top = 0;
        std::vector<double> w(size_t(K), 0.0);
        for (int32_t n = 0; n < N; n++) {
            for (int32_t k = 0; k < K; k++) {
                const size_t word = size_t(n) / 8, shift = size_t(4 * place[n % 8]), g = size_t(k) / 128;
                const int q = int(qw[size_t(k) * (N / 8) + word] >> shift) & 15, z = int(qz[g * (N / 8) + word] >> shift) & 15;
                w[size_t(k)] = (q - z) * (1.0 + (scales[g * N + size_t(n)] & 1023) / 1024.0) / 128.0;
            }
            for (int32_t m = 0; m < M; m++) {
                double sum = 0;
                for (int32_t k = 0; k < K; k++) sum += double(x[size_t(m) * K + size_t(k)]) * w[size_t(k)];
                worst = std::max(worst, std::abs(sum - double(y[size_t(m) * N + size_t(n)])));
                top = std::max(top, std::abs(sum));
            }
        }
        return worst / top;
    }
};

// a few rows through a layer that has not asked for any summation order: what the GEMV gives
void test_matmul_rows_cuda(Report& rep) {
    const double half = 1e-3;  // x rounded to fp16, 2^-12 per product on average
    {  // the GEMV's workspace alone
        QuantCase c(rep, 8, 256, 128);
        EXPECT(c.error(c.run(rep)) <= half);
        c.layer.set_accumulate(true);  // onto zeros
        EXPECT(c.error(c.run(rep)) <= half);
    }
    {  // a width the GEMV multiplies in fp32, weights as they are: K fp32 roundings
        QuantCase c(rep, 8, 256, 136);
        c.layer.set_gemm_workspace(QuantCase::scratch(kernel::matmul_quant_gemm_workspace_bytes(c.M, c.K)));
        EXPECT(c.error(c.run(rep)) <= 256 * 0x1p-24);
    }
    for (bool accumulate : {false, true}) {  // K in 32 groups: a sum of many partial sums
        QuantCase c(rep, 8, 4096, 512);
        c.layer.set_gemm_workspace(QuantCase::scratch(kernel::matmul_quant_gemm_workspace_bytes(c.M, c.K)));
        c.layer.set_accumulate(accumulate);
        const std::vector<float> first = c.run(rep);
        EXPECT(c.error(first) <= half);
        for (int i = 0; i < 10 && !accumulate; i++) EXPECT(c.run(rep) == first);  // the order is fixed
    }
    {  // 400 tiles of 128 x 256 rows and columns: large enough for whole tiles, whose order is fixed
        QuantCase c(rep, 2048, 1024, 6400);
        c.layer.set_gemm_workspace(QuantCase::scratch(kernel::matmul_quant_gemm_workspace_bytes(c.M, c.K)));
        const std::vector<float> first = c.run(rep);
        for (int i = 0; i < 3; i++) EXPECT(c.run(rep) == first);
    }
}

}  // namespace

extern "C" int kuiper_selftest(int use_cuda, char* report, size_t report_bytes) {
    Report rep;
    test_status(rep);
    test_buffer_cpu(rep);
    test_tensor_cpu(rep);
    test_layer_cpu(rep);
    if (use_cuda) {
        test_cuda(rep);
        test_matmul_rows_cuda(rep);
    }
    rep.out << rep.passed << " checks passed, " << rep.failed << " failed\n";
    if (report && report_bytes > 0) {
        const std::string s = rep.out.str();
        const size_t n = s.size() < report_bytes - 1 ? s.size() : report_bytes - 1;
        std::memcpy(report, s.data(), n);
        report[n] = '\0';
    }
    return rep.failed;
}
