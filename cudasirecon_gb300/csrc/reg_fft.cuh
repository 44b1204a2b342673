// Register-resident four-step FFT path for the shared-memory engine.
//
// A line of N = P * E points is held by P cooperating lanes of a warp, lane p
// holding x[p + P*e] (e < E) in registers.  Each lane runs an in-register DFT
// of length E (over e), multiplies by W_N^(p*k1), the lanes exchange once
// through a padded warp-private shared buffer ((P+1) x E, conflict-free), and
// each lane runs in-register DFTs of length P for k1 = p + P*m.  Lane p then
// holds X[p + P*m + E*k2] at v[m*P + k2].  One exchange per transform and
// only __syncwarp() -- no CTA barriers and no per-stage shared round trips.
//
// The compile-time DFTs split composite lengths recursively (N = A*B,
// inner DFT_B over x[i + A*j], twiddle W_N^(i*k1), outer DFT_A), with the
// twiddles taken from a table of W_480, or for lengths that do not divide 480
// from a table formed at compile time.
#pragma once
#include "fft.cuh"

namespace simrecon {

#ifdef __CUDACC__
__device__ __forceinline__ float2 w480c(int m, int dir)
{
  constexpr float c[480] = {
    1.000000000e+00f, 9.999143276e-01f, 9.996573250e-01f, 9.992290362e-01f, 9.986295348e-01f, 9.978589232e-01f,
    9.969173337e-01f, 9.958049276e-01f, 9.945218954e-01f, 9.930684570e-01f, 9.914448614e-01f, 9.896513868e-01f,
    9.876883406e-01f, 9.855560591e-01f, 9.832549076e-01f, 9.807852804e-01f, 9.781476007e-01f, 9.753423205e-01f,
    9.723699204e-01f, 9.692309097e-01f, 9.659258263e-01f, 9.624552365e-01f, 9.588197349e-01f, 9.550199445e-01f,
    9.510565163e-01f, 9.469301295e-01f, 9.426414911e-01f, 9.381913359e-01f, 9.335804265e-01f, 9.288095529e-01f,
    9.238795325e-01f, 9.187912101e-01f, 9.135454576e-01f, 9.081431738e-01f, 9.025852843e-01f, 8.968727415e-01f,
    8.910065242e-01f, 8.849876375e-01f, 8.788171127e-01f, 8.724960071e-01f, 8.660254038e-01f, 8.594064115e-01f,
    8.526401644e-01f, 8.457278217e-01f, 8.386705679e-01f, 8.314696123e-01f, 8.241261886e-01f, 8.166415552e-01f,
    8.090169944e-01f, 8.012538127e-01f, 7.933533403e-01f, 7.853169309e-01f, 7.771459615e-01f, 7.688418321e-01f,
    7.604059656e-01f, 7.518398075e-01f, 7.431448255e-01f, 7.343225094e-01f, 7.253743710e-01f, 7.163019434e-01f,
    7.071067812e-01f, 6.977904598e-01f, 6.883545757e-01f, 6.788007455e-01f, 6.691306064e-01f, 6.593458151e-01f,
    6.494480483e-01f, 6.394390020e-01f, 6.293203910e-01f, 6.190939493e-01f, 6.087614290e-01f, 5.983246006e-01f,
    5.877852523e-01f, 5.771451900e-01f, 5.664062369e-01f, 5.555702330e-01f, 5.446390350e-01f, 5.336145159e-01f,
    5.224985647e-01f, 5.112930861e-01f, 5.000000000e-01f, 4.886212415e-01f, 4.771587603e-01f, 4.656145203e-01f,
    4.539904997e-01f, 4.422886902e-01f, 4.305110968e-01f, 4.186597375e-01f, 4.067366431e-01f, 3.947438564e-01f,
    3.826834324e-01f, 3.705574375e-01f, 3.583679495e-01f, 3.461170571e-01f, 3.338068592e-01f, 3.214394653e-01f,
    3.090169944e-01f, 2.965415750e-01f, 2.840153447e-01f, 2.714404499e-01f, 2.588190451e-01f, 2.461532930e-01f,
    2.334453639e-01f, 2.206974350e-01f, 2.079116908e-01f, 1.950903220e-01f, 1.822355255e-01f, 1.693495038e-01f,
    1.564344650e-01f, 1.434926220e-01f, 1.305261922e-01f, 1.175373975e-01f, 1.045284633e-01f, 9.150161866e-02f,
    7.845909573e-02f, 6.540312923e-02f, 5.233595624e-02f, 3.925981576e-02f, 2.617694831e-02f, 1.308959557e-02f,
    2.832769449e-16f, -1.308959557e-02f, -2.617694831e-02f, -3.925981576e-02f, -5.233595624e-02f,
    -6.540312923e-02f, -7.845909573e-02f, -9.150161866e-02f, -1.045284633e-01f, -1.175373975e-01f,
    -1.305261922e-01f, -1.434926220e-01f, -1.564344650e-01f, -1.693495038e-01f, -1.822355255e-01f,
    -1.950903220e-01f, -2.079116908e-01f, -2.206974350e-01f, -2.334453639e-01f, -2.461532930e-01f,
    -2.588190451e-01f, -2.714404499e-01f, -2.840153447e-01f, -2.965415750e-01f, -3.090169944e-01f,
    -3.214394653e-01f, -3.338068592e-01f, -3.461170571e-01f, -3.583679495e-01f, -3.705574375e-01f,
    -3.826834324e-01f, -3.947438564e-01f, -4.067366431e-01f, -4.186597375e-01f, -4.305110968e-01f,
    -4.422886902e-01f, -4.539904997e-01f, -4.656145203e-01f, -4.771587603e-01f, -4.886212415e-01f,
    -5.000000000e-01f, -5.112930861e-01f, -5.224985647e-01f, -5.336145159e-01f, -5.446390350e-01f,
    -5.555702330e-01f, -5.664062369e-01f, -5.771451900e-01f, -5.877852523e-01f, -5.983246006e-01f,
    -6.087614290e-01f, -6.190939493e-01f, -6.293203910e-01f, -6.394390020e-01f, -6.494480483e-01f,
    -6.593458151e-01f, -6.691306064e-01f, -6.788007455e-01f, -6.883545757e-01f, -6.977904598e-01f,
    -7.071067812e-01f, -7.163019434e-01f, -7.253743710e-01f, -7.343225094e-01f, -7.431448255e-01f,
    -7.518398075e-01f, -7.604059656e-01f, -7.688418321e-01f, -7.771459615e-01f, -7.853169309e-01f,
    -7.933533403e-01f, -8.012538127e-01f, -8.090169944e-01f, -8.166415552e-01f, -8.241261886e-01f,
    -8.314696123e-01f, -8.386705679e-01f, -8.457278217e-01f, -8.526401644e-01f, -8.594064115e-01f,
    -8.660254038e-01f, -8.724960071e-01f, -8.788171127e-01f, -8.849876375e-01f, -8.910065242e-01f,
    -8.968727415e-01f, -9.025852843e-01f, -9.081431738e-01f, -9.135454576e-01f, -9.187912101e-01f,
    -9.238795325e-01f, -9.288095529e-01f, -9.335804265e-01f, -9.381913359e-01f, -9.426414911e-01f,
    -9.469301295e-01f, -9.510565163e-01f, -9.550199445e-01f, -9.588197349e-01f, -9.624552365e-01f,
    -9.659258263e-01f, -9.692309097e-01f, -9.723699204e-01f, -9.753423205e-01f, -9.781476007e-01f,
    -9.807852804e-01f, -9.832549076e-01f, -9.855560591e-01f, -9.876883406e-01f, -9.896513868e-01f,
    -9.914448614e-01f, -9.930684570e-01f, -9.945218954e-01f, -9.958049276e-01f, -9.969173337e-01f,
    -9.978589232e-01f, -9.986295348e-01f, -9.992290362e-01f, -9.996573250e-01f, -9.999143276e-01f,
    -1.000000000e+00f, -9.999143276e-01f, -9.996573250e-01f, -9.992290362e-01f, -9.986295348e-01f,
    -9.978589232e-01f, -9.969173337e-01f, -9.958049276e-01f, -9.945218954e-01f, -9.930684570e-01f,
    -9.914448614e-01f, -9.896513868e-01f, -9.876883406e-01f, -9.855560591e-01f, -9.832549076e-01f,
    -9.807852804e-01f, -9.781476007e-01f, -9.753423205e-01f, -9.723699204e-01f, -9.692309097e-01f,
    -9.659258263e-01f, -9.624552365e-01f, -9.588197349e-01f, -9.550199445e-01f, -9.510565163e-01f,
    -9.469301295e-01f, -9.426414911e-01f, -9.381913359e-01f, -9.335804265e-01f, -9.288095529e-01f,
    -9.238795325e-01f, -9.187912101e-01f, -9.135454576e-01f, -9.081431738e-01f, -9.025852843e-01f,
    -8.968727415e-01f, -8.910065242e-01f, -8.849876375e-01f, -8.788171127e-01f, -8.724960071e-01f,
    -8.660254038e-01f, -8.594064115e-01f, -8.526401644e-01f, -8.457278217e-01f, -8.386705679e-01f,
    -8.314696123e-01f, -8.241261886e-01f, -8.166415552e-01f, -8.090169944e-01f, -8.012538127e-01f,
    -7.933533403e-01f, -7.853169309e-01f, -7.771459615e-01f, -7.688418321e-01f, -7.604059656e-01f,
    -7.518398075e-01f, -7.431448255e-01f, -7.343225094e-01f, -7.253743710e-01f, -7.163019434e-01f,
    -7.071067812e-01f, -6.977904598e-01f, -6.883545757e-01f, -6.788007455e-01f, -6.691306064e-01f,
    -6.593458151e-01f, -6.494480483e-01f, -6.394390020e-01f, -6.293203910e-01f, -6.190939493e-01f,
    -6.087614290e-01f, -5.983246006e-01f, -5.877852523e-01f, -5.771451900e-01f, -5.664062369e-01f,
    -5.555702330e-01f, -5.446390350e-01f, -5.336145159e-01f, -5.224985647e-01f, -5.112930861e-01f,
    -5.000000000e-01f, -4.886212415e-01f, -4.771587603e-01f, -4.656145203e-01f, -4.539904997e-01f,
    -4.422886902e-01f, -4.305110968e-01f, -4.186597375e-01f, -4.067366431e-01f, -3.947438564e-01f,
    -3.826834324e-01f, -3.705574375e-01f, -3.583679495e-01f, -3.461170571e-01f, -3.338068592e-01f,
    -3.214394653e-01f, -3.090169944e-01f, -2.965415750e-01f, -2.840153447e-01f, -2.714404499e-01f,
    -2.588190451e-01f, -2.461532930e-01f, -2.334453639e-01f, -2.206974350e-01f, -2.079116908e-01f,
    -1.950903220e-01f, -1.822355255e-01f, -1.693495038e-01f, -1.564344650e-01f, -1.434926220e-01f,
    -1.305261922e-01f, -1.175373975e-01f, -1.045284633e-01f, -9.150161866e-02f, -7.845909573e-02f,
    -6.540312923e-02f, -5.233595624e-02f, -3.925981576e-02f, -2.617694831e-02f, -1.308959557e-02f,
    -1.836970199e-16f, 1.308959557e-02f, 2.617694831e-02f, 3.925981576e-02f, 5.233595624e-02f, 6.540312923e-02f,
    7.845909573e-02f, 9.150161866e-02f, 1.045284633e-01f, 1.175373975e-01f, 1.305261922e-01f, 1.434926220e-01f,
    1.564344650e-01f, 1.693495038e-01f, 1.822355255e-01f, 1.950903220e-01f, 2.079116908e-01f, 2.206974350e-01f,
    2.334453639e-01f, 2.461532930e-01f, 2.588190451e-01f, 2.714404499e-01f, 2.840153447e-01f, 2.965415750e-01f,
    3.090169944e-01f, 3.214394653e-01f, 3.338068592e-01f, 3.461170571e-01f, 3.583679495e-01f, 3.705574375e-01f,
    3.826834324e-01f, 3.947438564e-01f, 4.067366431e-01f, 4.186597375e-01f, 4.305110968e-01f, 4.422886902e-01f,
    4.539904997e-01f, 4.656145203e-01f, 4.771587603e-01f, 4.886212415e-01f, 5.000000000e-01f, 5.112930861e-01f,
    5.224985647e-01f, 5.336145159e-01f, 5.446390350e-01f, 5.555702330e-01f, 5.664062369e-01f, 5.771451900e-01f,
    5.877852523e-01f, 5.983246006e-01f, 6.087614290e-01f, 6.190939493e-01f, 6.293203910e-01f, 6.394390020e-01f,
    6.494480483e-01f, 6.593458151e-01f, 6.691306064e-01f, 6.788007455e-01f, 6.883545757e-01f, 6.977904598e-01f,
    7.071067812e-01f, 7.163019434e-01f, 7.253743710e-01f, 7.343225094e-01f, 7.431448255e-01f, 7.518398075e-01f,
    7.604059656e-01f, 7.688418321e-01f, 7.771459615e-01f, 7.853169309e-01f, 7.933533403e-01f, 8.012538127e-01f,
    8.090169944e-01f, 8.166415552e-01f, 8.241261886e-01f, 8.314696123e-01f, 8.386705679e-01f, 8.457278217e-01f,
    8.526401644e-01f, 8.594064115e-01f, 8.660254038e-01f, 8.724960071e-01f, 8.788171127e-01f, 8.849876375e-01f,
    8.910065242e-01f, 8.968727415e-01f, 9.025852843e-01f, 9.081431738e-01f, 9.135454576e-01f, 9.187912101e-01f,
    9.238795325e-01f, 9.288095529e-01f, 9.335804265e-01f, 9.381913359e-01f, 9.426414911e-01f, 9.469301295e-01f,
    9.510565163e-01f, 9.550199445e-01f, 9.588197349e-01f, 9.624552365e-01f, 9.659258263e-01f, 9.692309097e-01f,
    9.723699204e-01f, 9.753423205e-01f, 9.781476007e-01f, 9.807852804e-01f, 9.832549076e-01f, 9.855560591e-01f,
    9.876883406e-01f, 9.896513868e-01f, 9.914448614e-01f, 9.930684570e-01f, 9.945218954e-01f, 9.958049276e-01f,
    9.969173337e-01f, 9.978589232e-01f, 9.986295348e-01f, 9.992290362e-01f, 9.996573250e-01f, 9.999143276e-01f};
  constexpr float s[480] = {
    0.000000000e+00f, 1.308959557e-02f, 2.617694831e-02f, 3.925981576e-02f, 5.233595624e-02f, 6.540312923e-02f,
    7.845909573e-02f, 9.150161866e-02f, 1.045284633e-01f, 1.175373975e-01f, 1.305261922e-01f, 1.434926220e-01f,
    1.564344650e-01f, 1.693495038e-01f, 1.822355255e-01f, 1.950903220e-01f, 2.079116908e-01f, 2.206974350e-01f,
    2.334453639e-01f, 2.461532930e-01f, 2.588190451e-01f, 2.714404499e-01f, 2.840153447e-01f, 2.965415750e-01f,
    3.090169944e-01f, 3.214394653e-01f, 3.338068592e-01f, 3.461170571e-01f, 3.583679495e-01f, 3.705574375e-01f,
    3.826834324e-01f, 3.947438564e-01f, 4.067366431e-01f, 4.186597375e-01f, 4.305110968e-01f, 4.422886902e-01f,
    4.539904997e-01f, 4.656145203e-01f, 4.771587603e-01f, 4.886212415e-01f, 5.000000000e-01f, 5.112930861e-01f,
    5.224985647e-01f, 5.336145159e-01f, 5.446390350e-01f, 5.555702330e-01f, 5.664062369e-01f, 5.771451900e-01f,
    5.877852523e-01f, 5.983246006e-01f, 6.087614290e-01f, 6.190939493e-01f, 6.293203910e-01f, 6.394390020e-01f,
    6.494480483e-01f, 6.593458151e-01f, 6.691306064e-01f, 6.788007455e-01f, 6.883545757e-01f, 6.977904598e-01f,
    7.071067812e-01f, 7.163019434e-01f, 7.253743710e-01f, 7.343225094e-01f, 7.431448255e-01f, 7.518398075e-01f,
    7.604059656e-01f, 7.688418321e-01f, 7.771459615e-01f, 7.853169309e-01f, 7.933533403e-01f, 8.012538127e-01f,
    8.090169944e-01f, 8.166415552e-01f, 8.241261886e-01f, 8.314696123e-01f, 8.386705679e-01f, 8.457278217e-01f,
    8.526401644e-01f, 8.594064115e-01f, 8.660254038e-01f, 8.724960071e-01f, 8.788171127e-01f, 8.849876375e-01f,
    8.910065242e-01f, 8.968727415e-01f, 9.025852843e-01f, 9.081431738e-01f, 9.135454576e-01f, 9.187912101e-01f,
    9.238795325e-01f, 9.288095529e-01f, 9.335804265e-01f, 9.381913359e-01f, 9.426414911e-01f, 9.469301295e-01f,
    9.510565163e-01f, 9.550199445e-01f, 9.588197349e-01f, 9.624552365e-01f, 9.659258263e-01f, 9.692309097e-01f,
    9.723699204e-01f, 9.753423205e-01f, 9.781476007e-01f, 9.807852804e-01f, 9.832549076e-01f, 9.855560591e-01f,
    9.876883406e-01f, 9.896513868e-01f, 9.914448614e-01f, 9.930684570e-01f, 9.945218954e-01f, 9.958049276e-01f,
    9.969173337e-01f, 9.978589232e-01f, 9.986295348e-01f, 9.992290362e-01f, 9.996573250e-01f, 9.999143276e-01f,
    1.000000000e+00f, 9.999143276e-01f, 9.996573250e-01f, 9.992290362e-01f, 9.986295348e-01f, 9.978589232e-01f,
    9.969173337e-01f, 9.958049276e-01f, 9.945218954e-01f, 9.930684570e-01f, 9.914448614e-01f, 9.896513868e-01f,
    9.876883406e-01f, 9.855560591e-01f, 9.832549076e-01f, 9.807852804e-01f, 9.781476007e-01f, 9.753423205e-01f,
    9.723699204e-01f, 9.692309097e-01f, 9.659258263e-01f, 9.624552365e-01f, 9.588197349e-01f, 9.550199445e-01f,
    9.510565163e-01f, 9.469301295e-01f, 9.426414911e-01f, 9.381913359e-01f, 9.335804265e-01f, 9.288095529e-01f,
    9.238795325e-01f, 9.187912101e-01f, 9.135454576e-01f, 9.081431738e-01f, 9.025852843e-01f, 8.968727415e-01f,
    8.910065242e-01f, 8.849876375e-01f, 8.788171127e-01f, 8.724960071e-01f, 8.660254038e-01f, 8.594064115e-01f,
    8.526401644e-01f, 8.457278217e-01f, 8.386705679e-01f, 8.314696123e-01f, 8.241261886e-01f, 8.166415552e-01f,
    8.090169944e-01f, 8.012538127e-01f, 7.933533403e-01f, 7.853169309e-01f, 7.771459615e-01f, 7.688418321e-01f,
    7.604059656e-01f, 7.518398075e-01f, 7.431448255e-01f, 7.343225094e-01f, 7.253743710e-01f, 7.163019434e-01f,
    7.071067812e-01f, 6.977904598e-01f, 6.883545757e-01f, 6.788007455e-01f, 6.691306064e-01f, 6.593458151e-01f,
    6.494480483e-01f, 6.394390020e-01f, 6.293203910e-01f, 6.190939493e-01f, 6.087614290e-01f, 5.983246006e-01f,
    5.877852523e-01f, 5.771451900e-01f, 5.664062369e-01f, 5.555702330e-01f, 5.446390350e-01f, 5.336145159e-01f,
    5.224985647e-01f, 5.112930861e-01f, 5.000000000e-01f, 4.886212415e-01f, 4.771587603e-01f, 4.656145203e-01f,
    4.539904997e-01f, 4.422886902e-01f, 4.305110968e-01f, 4.186597375e-01f, 4.067366431e-01f, 3.947438564e-01f,
    3.826834324e-01f, 3.705574375e-01f, 3.583679495e-01f, 3.461170571e-01f, 3.338068592e-01f, 3.214394653e-01f,
    3.090169944e-01f, 2.965415750e-01f, 2.840153447e-01f, 2.714404499e-01f, 2.588190451e-01f, 2.461532930e-01f,
    2.334453639e-01f, 2.206974350e-01f, 2.079116908e-01f, 1.950903220e-01f, 1.822355255e-01f, 1.693495038e-01f,
    1.564344650e-01f, 1.434926220e-01f, 1.305261922e-01f, 1.175373975e-01f, 1.045284633e-01f, 9.150161866e-02f,
    7.845909573e-02f, 6.540312923e-02f, 5.233595624e-02f, 3.925981576e-02f, 2.617694831e-02f, 1.308959557e-02f,
    5.665538898e-16f, -1.308959557e-02f, -2.617694831e-02f, -3.925981576e-02f, -5.233595624e-02f,
    -6.540312923e-02f, -7.845909573e-02f, -9.150161866e-02f, -1.045284633e-01f, -1.175373975e-01f,
    -1.305261922e-01f, -1.434926220e-01f, -1.564344650e-01f, -1.693495038e-01f, -1.822355255e-01f,
    -1.950903220e-01f, -2.079116908e-01f, -2.206974350e-01f, -2.334453639e-01f, -2.461532930e-01f,
    -2.588190451e-01f, -2.714404499e-01f, -2.840153447e-01f, -2.965415750e-01f, -3.090169944e-01f,
    -3.214394653e-01f, -3.338068592e-01f, -3.461170571e-01f, -3.583679495e-01f, -3.705574375e-01f,
    -3.826834324e-01f, -3.947438564e-01f, -4.067366431e-01f, -4.186597375e-01f, -4.305110968e-01f,
    -4.422886902e-01f, -4.539904997e-01f, -4.656145203e-01f, -4.771587603e-01f, -4.886212415e-01f,
    -5.000000000e-01f, -5.112930861e-01f, -5.224985647e-01f, -5.336145159e-01f, -5.446390350e-01f,
    -5.555702330e-01f, -5.664062369e-01f, -5.771451900e-01f, -5.877852523e-01f, -5.983246006e-01f,
    -6.087614290e-01f, -6.190939493e-01f, -6.293203910e-01f, -6.394390020e-01f, -6.494480483e-01f,
    -6.593458151e-01f, -6.691306064e-01f, -6.788007455e-01f, -6.883545757e-01f, -6.977904598e-01f,
    -7.071067812e-01f, -7.163019434e-01f, -7.253743710e-01f, -7.343225094e-01f, -7.431448255e-01f,
    -7.518398075e-01f, -7.604059656e-01f, -7.688418321e-01f, -7.771459615e-01f, -7.853169309e-01f,
    -7.933533403e-01f, -8.012538127e-01f, -8.090169944e-01f, -8.166415552e-01f, -8.241261886e-01f,
    -8.314696123e-01f, -8.386705679e-01f, -8.457278217e-01f, -8.526401644e-01f, -8.594064115e-01f,
    -8.660254038e-01f, -8.724960071e-01f, -8.788171127e-01f, -8.849876375e-01f, -8.910065242e-01f,
    -8.968727415e-01f, -9.025852843e-01f, -9.081431738e-01f, -9.135454576e-01f, -9.187912101e-01f,
    -9.238795325e-01f, -9.288095529e-01f, -9.335804265e-01f, -9.381913359e-01f, -9.426414911e-01f,
    -9.469301295e-01f, -9.510565163e-01f, -9.550199445e-01f, -9.588197349e-01f, -9.624552365e-01f,
    -9.659258263e-01f, -9.692309097e-01f, -9.723699204e-01f, -9.753423205e-01f, -9.781476007e-01f,
    -9.807852804e-01f, -9.832549076e-01f, -9.855560591e-01f, -9.876883406e-01f, -9.896513868e-01f,
    -9.914448614e-01f, -9.930684570e-01f, -9.945218954e-01f, -9.958049276e-01f, -9.969173337e-01f,
    -9.978589232e-01f, -9.986295348e-01f, -9.992290362e-01f, -9.996573250e-01f, -9.999143276e-01f,
    -1.000000000e+00f, -9.999143276e-01f, -9.996573250e-01f, -9.992290362e-01f, -9.986295348e-01f,
    -9.978589232e-01f, -9.969173337e-01f, -9.958049276e-01f, -9.945218954e-01f, -9.930684570e-01f,
    -9.914448614e-01f, -9.896513868e-01f, -9.876883406e-01f, -9.855560591e-01f, -9.832549076e-01f,
    -9.807852804e-01f, -9.781476007e-01f, -9.753423205e-01f, -9.723699204e-01f, -9.692309097e-01f,
    -9.659258263e-01f, -9.624552365e-01f, -9.588197349e-01f, -9.550199445e-01f, -9.510565163e-01f,
    -9.469301295e-01f, -9.426414911e-01f, -9.381913359e-01f, -9.335804265e-01f, -9.288095529e-01f,
    -9.238795325e-01f, -9.187912101e-01f, -9.135454576e-01f, -9.081431738e-01f, -9.025852843e-01f,
    -8.968727415e-01f, -8.910065242e-01f, -8.849876375e-01f, -8.788171127e-01f, -8.724960071e-01f,
    -8.660254038e-01f, -8.594064115e-01f, -8.526401644e-01f, -8.457278217e-01f, -8.386705679e-01f,
    -8.314696123e-01f, -8.241261886e-01f, -8.166415552e-01f, -8.090169944e-01f, -8.012538127e-01f,
    -7.933533403e-01f, -7.853169309e-01f, -7.771459615e-01f, -7.688418321e-01f, -7.604059656e-01f,
    -7.518398075e-01f, -7.431448255e-01f, -7.343225094e-01f, -7.253743710e-01f, -7.163019434e-01f,
    -7.071067812e-01f, -6.977904598e-01f, -6.883545757e-01f, -6.788007455e-01f, -6.691306064e-01f,
    -6.593458151e-01f, -6.494480483e-01f, -6.394390020e-01f, -6.293203910e-01f, -6.190939493e-01f,
    -6.087614290e-01f, -5.983246006e-01f, -5.877852523e-01f, -5.771451900e-01f, -5.664062369e-01f,
    -5.555702330e-01f, -5.446390350e-01f, -5.336145159e-01f, -5.224985647e-01f, -5.112930861e-01f,
    -5.000000000e-01f, -4.886212415e-01f, -4.771587603e-01f, -4.656145203e-01f, -4.539904997e-01f,
    -4.422886902e-01f, -4.305110968e-01f, -4.186597375e-01f, -4.067366431e-01f, -3.947438564e-01f,
    -3.826834324e-01f, -3.705574375e-01f, -3.583679495e-01f, -3.461170571e-01f, -3.338068592e-01f,
    -3.214394653e-01f, -3.090169944e-01f, -2.965415750e-01f, -2.840153447e-01f, -2.714404499e-01f,
    -2.588190451e-01f, -2.461532930e-01f, -2.334453639e-01f, -2.206974350e-01f, -2.079116908e-01f,
    -1.950903220e-01f, -1.822355255e-01f, -1.693495038e-01f, -1.564344650e-01f, -1.434926220e-01f,
    -1.305261922e-01f, -1.175373975e-01f, -1.045284633e-01f, -9.150161866e-02f, -7.845909573e-02f,
    -6.540312923e-02f, -5.233595624e-02f, -3.925981576e-02f, -2.617694831e-02f, -1.308959557e-02f};
  m %= 480;
  return make_float2(c[m], dir < 0 ? -s[m] : s[m]);
}

// cos / sin of 2 pi m / N, formed by the compiler in double: the angle within
// an eighth of a turn of a multiple of a quarter turn, then its Taylor series
struct RootVal {
  double c, s;
};
__host__ __device__ constexpr RootVal root_val(long long m, long long N)
{
  m = ((m % N) + N) % N;
  const long long q = (4 * m + N / 2) / N;  // nearest quarter turn
  const double x = 6.283185307179586476925286766559 * (double)(4 * m - q * N) / (double)(4 * N);
  const double x2 = x * x;
  double c = 1.0, s = x, tc = 1.0, ts = x;
  for (int k = 1; k <= 10; ++k) {
    tc *= -x2 / (double)((2 * k - 1) * (2 * k));
    ts *= -x2 / (double)((2 * k) * (2 * k + 1));
    c += tc;
    s += ts;
  }
  switch (q & 3) {
    case 0: return RootVal{c, s};
    case 1: return RootVal{-s, c};
    case 2: return RootVal{-c, -s};
    default: return RootVal{s, -c};
  }
}
template <int N>
struct RootTable {
  float c[N], s[N];
  __host__ __device__ constexpr RootTable() : c{}, s{}
  {
    for (int m = 0; m < N; ++m) {
      const RootVal r = root_val(m, N);
      c[m] = (float)r.c;
      s[m] = (float)r.s;
    }
  }
};
// exp(dir * 2 pi i m / N) for a compile-time m
template <int N>
__device__ __forceinline__ float2 w_root(int m, int dir)
{
  if constexpr (480 % N == 0) {
    return w480c(m * (480 / N), dir);
  } else {
    constexpr RootTable<N> t;
    m %= N;
    return make_float2(t.c[m], dir < 0 ? -t.s[m] : t.s[m]);
  }
}

template <int N, int DIR>
__device__ __forceinline__ void reg_dft(float2* v)
{
  if constexpr (N == 1) {
  } else if constexpr (N == 2 || N == 3 || N == 4 || N == 5 || N == 7 || N == 8 || N == 16 || N == 32) {
    dftR<N, DIR>(v);
  } else {
    constexpr int A = (N % 4 == 0) ? 4 : ((N % 2 == 0) ? 2 : ((N % 3 == 0) ? 3 : ((N % 5 == 0) ? 5 : 7)));
    constexpr int B = N / A;
    float2 a[N];
#pragma unroll
    for (int i = 0; i < A; ++i) {
      float2 t[B];
#pragma unroll
      for (int j = 0; j < B; ++j) t[j] = v[i + A * j];
      reg_dft<B, DIR>(t);
#pragma unroll
      for (int k1 = 0; k1 < B; ++k1) a[i * B + k1] = (i * k1 == 0) ? t[k1] : cmul(t[k1], w_root<N>(i * k1, DIR));
    }
#pragma unroll
    for (int k1 = 0; k1 < B; ++k1) {
      float2 u[A];
#pragma unroll
      for (int i = 0; i < A; ++i) u[i] = a[i * B + k1];
      reg_dft<A, DIR>(u);
#pragma unroll
      for (int k2 = 0; k2 < A; ++k2) v[k1 + B * k2] = u[k2];
    }
  }
}

// One line by the P lanes of a group.  v: E = N/P values (in: x[p + P*e];
// out: v[m*P + k2] = X[p + P*m + E*k2]).  xb: group-private (P+1)*E buffer.
// twr: the plan's lane-major twiddles (FFTPlan::twr).
// Every lane of the warp must call this (it contains full-warp __syncwarp);
// lanes of inactive groups pass act = false and touch no memory.
template <int N, int P, int DIR>
__device__ __forceinline__ void reg_line(float2* v, int p, float2* xb, const float2* __restrict__ twr, bool act)
{
  constexpr int E = N / P;
  static_assert(E % P == 0, "lane count must divide the per-lane length");
  reg_dft<E, DIR>(v);
#pragma unroll
  for (int k1 = 1; k1 < E; ++k1) {
    float2 w = act ? __ldg(twr + (k1 - 1) * P + p) : make_float2(1.f, 0.f);
    if (DIR > 0) w.y = -w.y;
    v[k1] = cmul(v[k1], w);
  }
  if (act) {
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) xb[k1 * (P + 1) + p] = v[k1];
  }
  __syncwarp();
#pragma unroll
  for (int m = 0; m < E / P; ++m) {
    float2 u[P];
#pragma unroll
    for (int q = 0; q < P; ++q) u[q] = act ? xb[(p + P * m) * (P + 1) + q] : make_float2(0.f, 0.f);
    reg_dft<P, DIR>(u);
#pragma unroll
    for (int k2 = 0; k2 < P; ++k2) v[m * P + k2] = u[k2];
  }
  __syncwarp();
}

// nl lines held in shared buffer `a` (element (l, i) at a[l*ldl + i*ldi]) are
// transformed in place; `xbuf` is exchange scratch of
// reg_xbuf_elems(N, blockDim, nl) elements (one slot per group g < nl).  The
// whole CTA must call it.  The line loop has the same trip count in every
// thread so that the warp-wide syncs inside reg_line are reached by all 32
// lanes even when the warp's groups own different numbers of lines.
template <int N, int P, int DIR>
__device__ __forceinline__ void reg_lines(float2* a, float2* xbuf, int nl, int ldl, int ldi, const float2* twr)
{
  constexpr int E = N / P;
  const int p = threadIdx.x % P, g = threadIdx.x / P, ng = blockDim.x / P;
  float2* xb = xbuf + g * ((P + 1) * E + 1);  // used only while g < nl
  for (int base = 0; base < nl; base += ng) {
    const int l = base + g;
    const bool act = l < nl;
    float2 v[E];
    float2* line = a + (act ? l : 0) * ldl;
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = act ? line[(p + P * e) * ldi] : make_float2(0.f, 0.f);
    reg_line<N, P, DIR>(v, p, xb, twr, act);
    if (act) {
#pragma unroll
      for (int m = 0; m < E / P; ++m)
#pragma unroll
        for (int k2 = 0; k2 < P; ++k2) line[(p + P * m + E * k2) * ldi] = v[m * P + k2];
    }
  }
  __syncthreads();
}
#endif  // __CUDACC__

// Lengths with a register path and their lane counts (0: none).  Kernels are
// instantiated per length (registers are allocated for the largest path a
// kernel contains), so the list is kept to the lengths the workloads use.
__host__ __device__ constexpr int reg_fft_lanes(int n)
{
  return n == 32 ? 4 : n == 48 ? 4 : n == 64 ? 8 : n == 96 ? 4 : n == 128 ? 8 : n == 256 ? 16 : n == 512 ? 16
       : n == 1024 ? 32 : 0;
}
// X-macro over those lengths
#define SIMRECON_REG_SIZES(X) X(32) X(48) X(64) X(96) X(128) X(256) X(512) X(1024)

// exchange scratch (complex elements) reg_lines needs for `threads` threads
// transforming `lines` lines (only groups g < lines ever touch their slot)
__host__ __device__ constexpr int reg_xbuf_elems(int n, int threads, int lines)
{
  return reg_fft_lanes(n) ? ((threads / reg_fft_lanes(n)) < lines ? (threads / reg_fft_lanes(n)) : lines) *
                                ((reg_fft_lanes(n) + 1) * (n / reg_fft_lanes(n)) + 1)
                          : 0;
}

// shared bytes of a transform stage: buffer A (`elems` = lines x pitch) plus
// the second buffer (Stockham ping-pong or register-path exchange)
inline size_t fft_stage_smem(int n, int lines, int elems, int threads)
{
  size_t a = (size_t)elems;
  size_t b = (size_t)reg_xbuf_elems(n, threads, lines);
  return (a + (b > a ? b : a)) * sizeof(float2);
}

#ifdef __CUDACC__
// Transform of compile-time length NF with the register path, or (NF == 0)
// of any length with the Stockham stages.  Returns the buffer holding the
// result (a, or b for the Stockham path).  b must hold
// max(nl*pitch, reg_xbuf_elems(n, blockDim, nl)) elements.
template <int NF, int DIR>
__device__ __forceinline__ float2* fft_dispatch(float2* a, float2* b, const FFTPlan& pl, int nl, int ldl, int ldi)
{
  if constexpr (NF == 0) {
    return fft_lines<DIR>(a, b, pl, nl, ldl, ldi);
  } else {
    reg_lines<NF, reg_fft_lanes(NF), DIR>(a, b, nl, ldl, ldi, pl.twr);
    return a;
  }
}
#endif  // __CUDACC__

// Transform call sites.  Each can use the register path or the Stockham
// stages for lengths that have both; the register path needs more registers
// per thread (fewer resident warps), so the better choice depends on the
// kernel around the transform.
enum FftSite {
  kSiteIngestX = 0,   // k_ingest_x: rows of raw planes
  kSiteIngestY,       // k_fft_cols: y columns of the bands
  kSiteSeparateZ,     // k_separate: z lines
  kSiteOvlX,          // k_ovl_build_x: overlap rows
  kSiteOvlY,          // k_ovl_y_accum: overlap columns
  kSiteCorrRows,      // k_fft_rows: cross-correlation rows
  kSiteCorrCols,      // k_fft_cols2: cross-correlation columns
  kSiteAsmY,          // k_asm_y: zoomed y columns
  kSiteAsmX,          // k_asm_x: zoomed x rows
  kSiteAsmZ,          // k_asm_z: zoomed z lines
  kSiteMakeOtf,       // makeotf's 3D PSF transforms
  kSiteSelfTest,      // FFT-engine self test (always allowed)
  kNumFftSites
};
// true when `site` may use the register path for length n: the built-in
// choice, or the bit mask in SIMRECON_FFT_REGISTER_SITES (hex, bit = site)
// when that is set
bool reg_fft_site_enabled(FftSite site, int n);

// Host: call F.template operator()<NF>() with NF = n when n has a register
// path enabled at `site`, else NF = 0.
template <typename F>
inline void dispatch_fft_len(FftSite site, int n, F&& f)
{
  if (!reg_fft_site_enabled(site, n)) {
    f.template operator()<0>();
    return;
  }
  switch (n) {
#define SIMRECON_DISPATCH_CASE(N) \
  case N:                         \
    f.template operator()<N>();   \
    return;
    SIMRECON_REG_SIZES(SIMRECON_DISPATCH_CASE)
#undef SIMRECON_DISPATCH_CASE
    default:
      f.template operator()<0>();
  }
}

}  // namespace simrecon
