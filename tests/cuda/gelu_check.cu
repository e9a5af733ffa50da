// Evaluates the network's GELU and its derivative (pfc_b200/csrc/fno_gelu.cuh) on the
// GPU: FP32 values from the file argv[1], pairs (GELU, derivative) to argv[2].
#include <cstdio>
#include <vector>

#include "../../pfc_b200/csrc/fno_gelu.cuh"

__global__ void eval(const float* z, float2* out, int n) {
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		out[i] = make_float2(pfcg::gelu(z[i]), pfcg::gelu_d(z[i]));
}

int main(int argc, char** argv) {
	if (argc != 3) return 2;
	FILE* f = fopen(argv[1], "rb");
	if (!f) return 2;
	std::vector<float> z;
	float v;
	while (fread(&v, sizeof v, 1, f) == 1) z.push_back(v);
	fclose(f);
	const int n = (int)z.size();
	float* dz = nullptr;
	float2* dout = nullptr;
	std::vector<float2> out(n);
	if (cudaMalloc(&dz, sizeof(float) * n) != cudaSuccess || cudaMalloc(&dout, sizeof(float2) * n) != cudaSuccess) return 3;
	if (cudaMemcpy(dz, z.data(), sizeof(float) * n, cudaMemcpyHostToDevice) != cudaSuccess) return 3;
	eval<<<296, 256>>>(dz, dout, n);
	if (cudaMemcpy(out.data(), dout, sizeof(float2) * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
	f = fopen(argv[2], "wb");
	if (!f || fwrite(out.data(), sizeof(float2), n, f) != (size_t)n || fclose(f)) return 2;
	return 0;
}
