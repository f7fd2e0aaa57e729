// Row (x-direction) kernel instantiations for float.
#include "lines_dispatch.cuh"
namespace obl {
template cudaError_t launch_rows<float>(int, int, const RowArgs<float> &, cudaStream_t);
std::vector<std::vector<double>> plan_tables(int n)
{
    switch (n) {
#define OBL_CASE(N) case N: return plan_tables_n<N>();
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return {};
}
bool line_length_supported(int n)
{
    switch (n) {
#define OBL_CASE(N) case N: return true;
        OBL_FOR_EACH_N(OBL_CASE)
#undef OBL_CASE
    }
    return false;
}
}
