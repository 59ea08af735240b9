// Specialised fused-elementwise programs.  GENERATED by gen_vm_static.py from the launch plans of the benchmark
// programs; regenerate after changing the planner's code generation.
#pragma once
namespace b2x {
// reduce:%5
template <> struct VmStatic<1> {
  static constexpr int n = 1;
  static constexpr unsigned long long hash = 17957204132566544674ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[1] = {{1, 2, 0, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[1] = {10}; return e[t]; }
};
// reduce:%5
template <> struct VmStatic<2> {
  static constexpr int n = 1;
  static constexpr unsigned long long hash = 17957205232078172885ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[1] = {{1, 2, 0, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[1] = {11}; return e[t]; }
};
// dot_general:%25
template <> struct VmStatic<3> {
  static constexpr int n = 2;
  static constexpr unsigned long long hash = 13793836619330337276ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[2] = {{1, 5, 0, 0, 0, 0}, {3, 2, 0, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[1] = {11}; return e[t]; }
};
// dot_general:%0
template <> struct VmStatic<4> {
  static constexpr int n = 2;
  static constexpr unsigned long long hash = 13793837718841965487ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[2] = {{1, 5, 0, 0, 0, 0}, {3, 2, 0, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[1] = {10}; return e[t]; }
};
// dot_general:%0
template <> struct VmStatic<5> {
  static constexpr int n = 2;
  static constexpr unsigned long long hash = 13793838818353593698ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[2] = {{1, 5, 0, 0, 0, 0}, {3, 2, 0, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[1] = {9}; return e[t]; }
};
// fused:stablehlo.multiply:%2
template <> struct VmStatic<6> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 6245108412357681216ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 2, 0, 0, 0, 0}, {7, 2, 1, 0, 0, 0}, {3, 2, 2, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[3] = {11, 11, 11}; return e[t]; }
};
// fused:stablehlo.multiply:%2
template <> struct VmStatic<7> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 6872148898644938981ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 2, 0, 0, 0, 0}, {7, 2, 1, 0, 0, 0}, {3, 2, 2, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[3] = {10, 10, 10}; return e[t]; }
};
// dot_general:%0+epilogue(%2 )
template <> struct VmStatic<8> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 9785095952354713316ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 5, 0, 0, 0, 0}, {4, 2, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {11, 11}; return e[t]; }
};
// fused:stablehlo.add:%1
template <> struct VmStatic<9> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 11047972838744394022ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 2, 0, 0, 0, 0}, {4, 2, 1, 0, 0, 0}, {3, 2, 2, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[3] = {10, 10, 10}; return e[t]; }
};
// fused:stablehlo.add:%1
template <> struct VmStatic<10> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 11675004528938626099ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 2, 0, 0, 0, 0}, {4, 2, 1, 0, 0, 0}, {3, 2, 2, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[3] = {11, 11, 11}; return e[t]; }
};
// fused:stablehlo.multiply:%60
template <> struct VmStatic<11> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 11988508811349373551ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 2, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {11, 11}; return e[t]; }
};
// fused:stablehlo.multiply:%4
template <> struct VmStatic<12> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 11989486277186663905ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 2, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {10, 10}; return e[t]; }
};
// dot_general:%25+epilogue(%57#1_scaled )
template <> struct VmStatic<13> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 17712653700945622981ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 5, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {3, 2, 0, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[1] = {11}; return e[t]; }
};
// reduce:%19+epilogue(%21 )
template <> struct VmStatic<14> {
  static constexpr int n = 3;
  static constexpr unsigned long long hash = 17972027340921337553ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[3] = {{1, 2, 0, 0, 0, 0}, {2, 0, 0, 0, 0, 0}, {7, 1, 0, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[1] = {11}; return e[t]; }
};
// dot_general:%0+epilogue(%3 )
template <> struct VmStatic<15> {
  static constexpr int n = 4;
  static constexpr unsigned long long hash = 14122777069394952415ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[4] = {{1, 5, 0, 0, 0, 0}, {4, 2, 0, 0, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {11, 10}; return e[t]; }
};
// dot_general:%0+epilogue(%4 )
template <> struct VmStatic<16> {
  static constexpr int n = 5;
  static constexpr unsigned long long hash = 2601592904018748018ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[5] = {{1, 5, 0, 0, 0, 0}, {4, 2, 0, 0, 0, 0}, {23, 0, 0, 1, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {11, 10}; return e[t]; }
};
// dot_general:%0+epilogue(%5 )
template <> struct VmStatic<17> {
  static constexpr int n = 5;
  static constexpr unsigned long long hash = 12980845326986873047ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[5] = {{1, 5, 0, 0, 0, 0}, {4, 2, 0, 0, 0, 0}, {10, 3, 0, 0, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {11, 10}; return e[t]; }
};
// dot_general:%0+epilogue(%4 )
template <> struct VmStatic<18> {
  static constexpr int n = 5;
  static constexpr unsigned long long hash = 16796294983129149687ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[5] = {{1, 5, 0, 0, 0, 0}, {4, 2, 0, 0, 0, 0}, {28, 0, 0, 1, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {11, 10}; return e[t]; }
};
// fused:stablehlo.convert:%3
template <> struct VmStatic<19> {
  static constexpr int n = 5;
  static constexpr unsigned long long hash = 17611560754473556635ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[5] = {{1, 2, 0, 0, 0, 0}, {4, 2, 1, 0, 0, 0}, {23, 0, 0, 1, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 2, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[3] = {11, 11, 10}; return e[t]; }
};
// dot_general:%16+epilogue(%24 )
template <> struct VmStatic<20> {
  static constexpr int n = 6;
  static constexpr unsigned long long hash = 7866583465631875640ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[6] = {{1, 5, 0, 0, 0, 0}, {3, 2, 0, 0, 0, 0}, {1, 5, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {11, 10}; return e[t]; }
};
// dot_general:%0+epilogue(%1 %15 )
template <> struct VmStatic<21> {
  static constexpr int n = 17;
  static constexpr unsigned long long hash = 5995960292406058526ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[17] = {{1, 5, 0, 0, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 0, 0, 0, 0}, {1, 5, 0, 0, 0, 0}, {7, 5, 0, 0, 0, 0}, {7, 5, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {4, 5, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {23, 0, 0, 0, 0, 0}, {4, 3, 0, 0, 0, 0}, {2, 0, 0, 0, 0, 0}, {1, 3, 0, 0, 0, 0}, {7, 5, 0, 0, 0, 0}, {7, 1, 0, 0, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {10, 10}; return e[t]; }
};
// dot_general:%0+epilogue(%16 )
template <> struct VmStatic<22> {
  static constexpr int n = 19;
  static constexpr unsigned long long hash = 1261296141604760860ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[19] = {{1, 5, 0, 0, 0, 0}, {4, 2, 0, 0, 0, 0}, {2, 0, 0, 0, 0, 0}, {1, 1, 0, 0, 0, 0}, {7, 1, 0, 0, 0, 0}, {7, 1, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {2, 0, 0, 1, 0, 0}, {1, 1, 0, 0, 0, 0}, {4, 1, 1, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {23, 0, 0, 1, 0, 0}, {4, 3, 0, 0, 0, 0}, {2, 0, 0, 1, 0, 0}, {1, 3, 0, 0, 0, 0}, {7, 1, 0, 0, 0, 0}, {7, 1, 1, 0, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {11, 10}; return e[t]; }
};
// dot_general:%26+epilogue(%55 )
template <> struct VmStatic<23> {
  static constexpr int n = 32;
  static constexpr unsigned long long hash = 649184291706289115ull;
  __host__ __device__ static constexpr VmSig at(int i) { constexpr VmSig c[32] = {{1, 2, 0, 0, 0, 0}, {2, 0, 0, 0, 0, 0}, {1, 1, 0, 0, 0, 0}, {7, 1, 0, 0, 0, 0}, {2, 0, 0, 1, 0, 0}, {7, 3, 0, 0, 0, 0}, {4, 3, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {2, 0, 0, 2, 0, 0}, {1, 1, 1, 0, 0, 0}, {7, 1, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {4, 1, 0, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {23, 0, 0, 0, 0, 0}, {2, 0, 0, 1, 0, 0}, {1, 1, 1, 0, 0, 0}, {7, 1, 1, 0, 0, 0}, {6, 3, 0, 0, 0, 0}, {2, 0, 0, 3, 0, 0}, {1, 3, 0, 0, 0, 0}, {7, 1, 0, 0, 0, 0}, {7, 1, 3, 0, 0, 0}, {7, 1, 2, 0, 0, 0}, {2, 0, 0, 2, 0, 0}, {1, 3, 0, 0, 0, 0}, {4, 1, 1, 0, 0, 0}, {7, 3, 0, 0, 0, 0}, {4, 1, 2, 0, 0, 0}, {7, 5, 0, 0, 0, 0}, {37, 0, 0, 0, 0, 0}, {3, 2, 1, 0, 0, 0}}; return c[i]; }
  __host__ __device__ static constexpr uint8_t elem(int t) { constexpr uint8_t e[2] = {10, 10}; return e[t]; }
};
__host__ inline int vm_static_lookup(uint64_t h) {
  switch (h) {
    case 17957204132566544674ull: return 1;
    case 17957205232078172885ull: return 2;
    case 13793836619330337276ull: return 3;
    case 13793837718841965487ull: return 4;
    case 13793838818353593698ull: return 5;
    case 6245108412357681216ull: return 6;
    case 6872148898644938981ull: return 7;
    case 9785095952354713316ull: return 8;
    case 11047972838744394022ull: return 9;
    case 11675004528938626099ull: return 10;
    case 11988508811349373551ull: return 11;
    case 11989486277186663905ull: return 12;
    case 17712653700945622981ull: return 13;
    case 17972027340921337553ull: return 14;
    case 14122777069394952415ull: return 15;
    case 2601592904018748018ull: return 16;
    case 12980845326986873047ull: return 17;
    case 16796294983129149687ull: return 18;
    case 17611560754473556635ull: return 19;
    case 7866583465631875640ull: return 20;
    case 5995960292406058526ull: return 21;
    case 1261296141604760860ull: return 22;
    case 649184291706289115ull: return 23;
    default: return 0;
  }
}
}  // namespace b2x
#define B2X_VM_STATIC_ELEMENTWISE(X) X(6) X(7) X(9) X(10) X(11) X(12) X(19)
#define B2X_VM_STATIC_REDUCE(X) X(1) X(2) X(14)
#define B2X_VM_STATIC_GEMM(X) X(3, 64) X(3, 128) X(3, 256) X(4, 64) X(4, 128) X(4, 256) X(5, 64) X(5, 128) X(5, 256) X(8, 64) X(8, 128) X(8, 256) X(13, 64) X(13, 128) X(13, 256) X(15, 64) X(15, 128) X(15, 256) X(16, 64) X(16, 128) X(16, 256) X(17, 64) X(17, 128) X(17, 256) X(18, 64) X(18, 128) X(18, 256) X(20, 64) X(20, 128) X(20, 256) X(21, 64) X(21, 128) X(21, 256) X(22, 64) X(22, 128) X(22, 256) X(23, 64) X(23, 128) X(23, 256)
