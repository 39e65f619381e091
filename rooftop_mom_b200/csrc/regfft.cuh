// Register-resident transforms of lines of n = n1 n2 points (device code only), n1 >= n2 both codelet lengths of
// at most 36. 12, 15 and every 7-smooth length from 16 to 1024 but 343, 686, 882 and 1000 have such a split; a length with
// a larger prime factor from 17 to 512 runs as a Bluestein convolution on a length m = n1 n2 >= 2 n - 1, the others take
// the Stockham engine of fft.cuh (make_reg_plan, runtime.cpp).
//
// The four-step form: thread t < n2 of a line holds x[n2 m1 + t] (the "A" layout),
//   reg_a_fwd: n1-point DFT over m1 in registers, twiddle w^(t k1), written to buf(k1, t);
//   reg_b_fwd: thread k1 < n1 reads row k1, n2-point DFT: X[k1 + n1 k2] (the "B" layout).
// The inverse runs the steps backwards, from the B layout to the A layout. Two exchanges through shared memory
// and two CTA barriers a transform, whatever the factors, against two barriers for every prime factor of the
// Stockham stages; the lengths are compile-time constants in each case of a switch on n1 or n2, so the
// butterflies stay in registers and the codelets' roots are constants.
#pragma once

#include <type_traits>

#include "fft.cuh"

namespace rtm {

// cos(2 pi k / R), 0 <= k <= R / 2.
template <int R> __host__ __device__ constexpr double root_cos_half(int k) {
    if constexpr (R == 3) {
        switch (k) { case 0: return 1.0; case 1: return -0.5; default: return 0; }
    } else if constexpr (R == 5) {
        switch (k) { case 0: return 1.0; case 1: return 0.30901699437494745; case 2: return -0.8090169943749475;
        default: return 0; }
    } else if constexpr (R == 6) {
        switch (k) { case 0: return 1.0; case 1: return 0.5; case 2: return -0.5; case 3: return -1.0; default:
        return 0; }
    } else if constexpr (R == 7) {
        switch (k) { case 0: return 1.0; case 1: return 0.6234898018587335; case 2: return -0.2225209339563144; case
        3: return -0.9009688679024191; default: return 0; }
    } else if constexpr (R == 9) {
        switch (k) { case 0: return 1.0; case 1: return 0.766044443118978; case 2: return 0.17364817766693036; case
        3: return -0.5; case 4: return -0.9396926207859084; default: return 0; }
    } else if constexpr (R == 10) {
        switch (k) { case 0: return 1.0; case 1: return 0.8090169943749475; case 2: return 0.30901699437494745; case
        3: return -0.30901699437494745; case 4: return -0.8090169943749475; case 5: return -1.0; default: return 0;
        }
    } else if constexpr (R == 12) {
        switch (k) { case 0: return 1.0; case 1: return 0.8660254037844386; case 2: return 0.5; case 3: return 0.0;
        case 4: return -0.5; case 5: return -0.8660254037844386; case 6: return -1.0; default: return 0; }
    } else if constexpr (R == 14) {
        switch (k) { case 0: return 1.0; case 1: return 0.9009688679024191; case 2: return 0.6234898018587335; case
        3: return 0.2225209339563144; case 4: return -0.2225209339563144; case 5: return -0.6234898018587335; case
        6: return -0.9009688679024191; case 7: return -1.0; default: return 0; }
    } else if constexpr (R == 15) {
        switch (k) { case 0: return 1.0; case 1: return 0.9135454576426009; case 2: return 0.6691306063588582; case
        3: return 0.30901699437494745; case 4: return -0.10452846326765347; case 5: return -0.5; case 6: return
        -0.8090169943749475; case 7: return -0.9781476007338057; default: return 0; }
    } else if constexpr (R == 18) {
        switch (k) { case 0: return 1.0; case 1: return 0.9396926207859084; case 2: return 0.766044443118978; case
        3: return 0.5; case 4: return 0.17364817766693036; case 5: return -0.17364817766693036; case 6: return -0.5;
        case 7: return -0.766044443118978; case 8: return -0.9396926207859084; case 9: return -1.0; default: return
        0; }
    } else if constexpr (R == 20) {
        switch (k) { case 0: return 1.0; case 1: return 0.9510565162951535; case 2: return 0.8090169943749475; case
        3: return 0.5877852522924731; case 4: return 0.30901699437494745; case 5: return 0.0; case 6: return
        -0.30901699437494745; case 7: return -0.5877852522924731; case 8: return -0.8090169943749475; case 9: return
        -0.9510565162951535; case 10: return -1.0; default: return 0; }
    } else if constexpr (R == 21) {
        switch (k) { case 0: return 1.0; case 1: return 0.9555728057861407; case 2: return 0.8262387743159949; case
        3: return 0.6234898018587335; case 4: return 0.36534102436639504; case 5: return 0.07473009358642425; case
        6: return -0.2225209339563144; case 7: return -0.5; case 8: return -0.7330518718298263; case 9: return
        -0.9009688679024191; case 10: return -0.9888308262251285; default: return 0; }
    } else if constexpr (R == 24) {
        switch (k) { case 0: return 1.0; case 1: return 0.9659258262890683; case 2: return 0.8660254037844386; case
        3: return 0.7071067811865476; case 4: return 0.5; case 5: return 0.25881904510252074; case 6: return 0.0;
        case 7: return -0.25881904510252074; case 8: return -0.5; case 9: return -0.7071067811865476; case 10:
        return -0.8660254037844386; case 11: return -0.9659258262890683; case 12: return -1.0; default: return 0; }
    } else if constexpr (R == 25) {
        switch (k) { case 0: return 1.0; case 1: return 0.9685831611286311; case 2: return 0.8763066800438636; case
        3: return 0.7289686274214116; case 4: return 0.5358267949789967; case 5: return 0.30901699437494745; case 6:
        return 0.06279051952931337; case 7: return -0.18738131458572463; case 8: return -0.42577929156507266; case
        9: return -0.6374239897486897; case 10: return -0.8090169943749475; case 11: return -0.9297764858882515;
        case 12: return -0.9921147013144779; default: return 0; }
    } else if constexpr (R == 27) {
        switch (k) { case 0: return 1.0; case 1: return 0.9730448705798238; case 2: return 0.8936326403234123; case
        3: return 0.766044443118978; case 4: return 0.5971585917027862; case 5: return 0.39607976603915684; case 6:
        return 0.17364817766693036; case 7: return -0.05814482891047583; case 8: return -0.28680323271109026; case
        9: return -0.5; case 10: return -0.6862416378687336; case 11: return -0.8354878114129364; case 12: return
        -0.9396926207859084; case 13: return -0.993238357741943; default: return 0; }
    } else if constexpr (R == 28) {
        switch (k) { case 0: return 1.0; case 1: return 0.9749279121818236; case 2: return 0.9009688679024191; case
        3: return 0.7818314824680298; case 4: return 0.6234898018587335; case 5: return 0.4338837391175581; case 6:
        return 0.2225209339563144; case 7: return 0.0; case 8: return -0.2225209339563144; case 9: return
        -0.4338837391175581; case 10: return -0.6234898018587335; case 11: return -0.7818314824680298; case 12:
        return -0.9009688679024191; case 13: return -0.9749279121818236; case 14: return -1.0; default: return 0; }
    } else if constexpr (R == 30) {
        switch (k) { case 0: return 1.0; case 1: return 0.9781476007338057; case 2: return 0.9135454576426009; case
        3: return 0.8090169943749475; case 4: return 0.6691306063588582; case 5: return 0.5; case 6: return
        0.30901699437494745; case 7: return 0.10452846326765347; case 8: return -0.10452846326765347; case 9: return
        -0.30901699437494745; case 10: return -0.5; case 11: return -0.6691306063588582; case 12: return
        -0.8090169943749475; case 13: return -0.9135454576426009; case 14: return -0.9781476007338057; case 15:
        return -1.0; default: return 0; }
    } else if constexpr (R == 32) {
        switch (k) { case 0: return 1.0; case 1: return 0.9807852804032304; case 2: return 0.9238795325112867; case
        3: return 0.8314696123025452; case 4: return 0.7071067811865476; case 5: return 0.5555702330196022; case 6:
        return 0.3826834323650898; case 7: return 0.19509032201612828; case 8: return 0.0; case 9: return
        -0.19509032201612828; case 10: return -0.3826834323650898; case 11: return -0.5555702330196022; case 12:
        return -0.7071067811865476; case 13: return -0.8314696123025452; case 14: return -0.9238795325112867; case
        15: return -0.9807852804032304; case 16: return -1.0; default: return 0; }
    } else if constexpr (R == 35) {
        switch (k) { case 0: return 1.0; case 1: return 0.9839295885986297; case 2: return 0.9362348706397372; case
        3: return 0.8584487936018661; case 4: return 0.753071466003611; case 5: return 0.6234898018587335; case 6:
        return 0.4738686624729987; case 7: return 0.30901699437494745; case 8: return 0.1342332658176555; case 9:
        return -0.044864830350514924; case 10: return -0.2225209339563144; case 11: return -0.3930250316539236; case
        12: return -0.5508969814521025; case 13: return -0.6910626489868646; case 14: return -0.8090169943749475;
        case 15: return -0.9009688679024191; case 16: return -0.9639628606958532; case 17: return
        -0.9959742939952391; default: return 0; }
    } else if constexpr (R == 36) {
        switch (k) { case 0: return 1.0; case 1: return 0.984807753012208; case 2: return 0.9396926207859084; case
        3: return 0.8660254037844386; case 4: return 0.766044443118978; case 5: return 0.6427876096865394; case 6:
        return 0.5; case 7: return 0.3420201433256687; case 8: return 0.17364817766693036; case 9: return 0.0; case
        10: return -0.17364817766693036; case 11: return -0.3420201433256687; case 12: return -0.5; case 13: return
        -0.6427876096865394; case 14: return -0.766044443118978; case 15: return -0.8660254037844386; case 16:
        return -0.9396926207859084; case 17: return -0.984807753012208; case 18: return -1.0; default: return 0; }
    }
    return 0;
}
// sin(2 pi k / R), 0 <= k <= R / 2.
template <int R> __host__ __device__ constexpr double root_sin_half(int k) {
    if constexpr (R == 3) {
        switch (k) { case 0: return 0.0; case 1: return 0.8660254037844386; default: return 0; }
    } else if constexpr (R == 5) {
        switch (k) { case 0: return 0.0; case 1: return 0.9510565162951535; case 2: return 0.5877852522924731;
        default: return 0; }
    } else if constexpr (R == 6) {
        switch (k) { case 0: return 0.0; case 1: return 0.8660254037844386; case 2: return 0.8660254037844386; case
        3: return 0.0; default: return 0; }
    } else if constexpr (R == 7) {
        switch (k) { case 0: return 0.0; case 1: return 0.7818314824680298; case 2: return 0.9749279121818236; case
        3: return 0.4338837391175581; default: return 0; }
    } else if constexpr (R == 9) {
        switch (k) { case 0: return 0.0; case 1: return 0.6427876096865394; case 2: return 0.984807753012208; case
        3: return 0.8660254037844386; case 4: return 0.3420201433256687; default: return 0; }
    } else if constexpr (R == 10) {
        switch (k) { case 0: return 0.0; case 1: return 0.5877852522924731; case 2: return 0.9510565162951535; case
        3: return 0.9510565162951535; case 4: return 0.5877852522924731; case 5: return 0.0; default: return 0; }
    } else if constexpr (R == 12) {
        switch (k) { case 0: return 0.0; case 1: return 0.5; case 2: return 0.8660254037844386; case 3: return 1.0;
        case 4: return 0.8660254037844386; case 5: return 0.5; case 6: return 0.0; default: return 0; }
    } else if constexpr (R == 14) {
        switch (k) { case 0: return 0.0; case 1: return 0.4338837391175581; case 2: return 0.7818314824680298; case
        3: return 0.9749279121818236; case 4: return 0.9749279121818236; case 5: return 0.7818314824680298; case 6:
        return 0.4338837391175581; case 7: return 0.0; default: return 0; }
    } else if constexpr (R == 15) {
        switch (k) { case 0: return 0.0; case 1: return 0.4067366430758002; case 2: return 0.7431448254773942; case
        3: return 0.9510565162951535; case 4: return 0.9945218953682733; case 5: return 0.8660254037844386; case 6:
        return 0.5877852522924731; case 7: return 0.20791169081775934; default: return 0; }
    } else if constexpr (R == 18) {
        switch (k) { case 0: return 0.0; case 1: return 0.3420201433256687; case 2: return 0.6427876096865394; case
        3: return 0.8660254037844386; case 4: return 0.984807753012208; case 5: return 0.984807753012208; case 6:
        return 0.8660254037844386; case 7: return 0.6427876096865394; case 8: return 0.3420201433256687; case 9:
        return 0.0; default: return 0; }
    } else if constexpr (R == 20) {
        switch (k) { case 0: return 0.0; case 1: return 0.30901699437494745; case 2: return 0.5877852522924731; case
        3: return 0.8090169943749475; case 4: return 0.9510565162951535; case 5: return 1.0; case 6: return
        0.9510565162951535; case 7: return 0.8090169943749475; case 8: return 0.5877852522924731; case 9: return
        0.30901699437494745; case 10: return 0.0; default: return 0; }
    } else if constexpr (R == 21) {
        switch (k) { case 0: return 0.0; case 1: return 0.2947551744109042; case 2: return 0.5633200580636221; case
        3: return 0.7818314824680298; case 4: return 0.9308737486442042; case 5: return 0.9972037971811801; case 6:
        return 0.9749279121818236; case 7: return 0.8660254037844386; case 8: return 0.6801727377709194; case 9:
        return 0.4338837391175581; case 10: return 0.14904226617617444; default: return 0; }
    } else if constexpr (R == 24) {
        switch (k) { case 0: return 0.0; case 1: return 0.25881904510252074; case 2: return 0.5; case 3: return
        0.7071067811865476; case 4: return 0.8660254037844386; case 5: return 0.9659258262890683; case 6: return
        1.0; case 7: return 0.9659258262890683; case 8: return 0.8660254037844386; case 9: return
        0.7071067811865476; case 10: return 0.5; case 11: return 0.25881904510252074; case 12: return 0.0; default:
        return 0; }
    } else if constexpr (R == 25) {
        switch (k) { case 0: return 0.0; case 1: return 0.2486898871648548; case 2: return 0.48175367410171527; case
        3: return 0.6845471059286887; case 4: return 0.8443279255020151; case 5: return 0.9510565162951535; case 6:
        return 0.9980267284282716; case 7: return 0.9822872507286887; case 8: return 0.9048270524660196; case 9:
        return 0.7705132427757893; case 10: return 0.5877852522924731; case 11: return 0.368124552684678; case 12:
        return 0.12533323356430426; default: return 0; }
    } else if constexpr (R == 27) {
        switch (k) { case 0: return 0.0; case 1: return 0.23061587074244017; case 2: return 0.44879918020046217;
        case 3: return 0.6427876096865394; case 4: return 0.8021231927550437; case 5: return 0.918216106880274; case
        6: return 0.984807753012208; case 7: return 0.9983081582712682; case 8: return 0.9579895123154889; case 9:
        return 0.8660254037844386; case 10: return 0.7273736415730487; case 11: return 0.549508978070806; case 12:
        return 0.3420201433256687; case 13: return 0.11609291412523023; default: return 0; }
    } else if constexpr (R == 28) {
        switch (k) { case 0: return 0.0; case 1: return 0.2225209339563144; case 2: return 0.4338837391175581; case
        3: return 0.6234898018587335; case 4: return 0.7818314824680298; case 5: return 0.9009688679024191; case 6:
        return 0.9749279121818236; case 7: return 1.0; case 8: return 0.9749279121818236; case 9: return
        0.9009688679024191; case 10: return 0.7818314824680298; case 11: return 0.6234898018587335; case 12: return
        0.4338837391175581; case 13: return 0.2225209339563144; case 14: return 0.0; default: return 0; }
    } else if constexpr (R == 30) {
        switch (k) { case 0: return 0.0; case 1: return 0.20791169081775934; case 2: return 0.4067366430758002; case
        3: return 0.5877852522924731; case 4: return 0.7431448254773942; case 5: return 0.8660254037844386; case 6:
        return 0.9510565162951535; case 7: return 0.9945218953682733; case 8: return 0.9945218953682733; case 9:
        return 0.9510565162951535; case 10: return 0.8660254037844386; case 11: return 0.7431448254773942; case 12:
        return 0.5877852522924731; case 13: return 0.4067366430758002; case 14: return 0.20791169081775934; case 15:
        return 0.0; default: return 0; }
    } else if constexpr (R == 32) {
        switch (k) { case 0: return 0.0; case 1: return 0.19509032201612828; case 2: return 0.3826834323650898; case
        3: return 0.5555702330196022; case 4: return 0.7071067811865476; case 5: return 0.8314696123025452; case 6:
        return 0.9238795325112867; case 7: return 0.9807852804032304; case 8: return 1.0; case 9: return
        0.9807852804032304; case 10: return 0.9238795325112867; case 11: return 0.8314696123025452; case 12: return
        0.7071067811865476; case 13: return 0.5555702330196022; case 14: return 0.3826834323650898; case 15: return
        0.19509032201612828; case 16: return 0.0; default: return 0; }
    } else if constexpr (R == 35) {
        switch (k) { case 0: return 0.0; case 1: return 0.17855689479863665; case 2: return 0.3513748240813427; case
        3: return 0.5128992774059061; case 4: return 0.6579387259397126; case 5: return 0.7818314824680298; case 6:
        return 0.880595531856738; case 7: return 0.9510565162951535; case 8: return 0.9909497617679347; case 9:
        return 0.9989930665413147; case 10: return 0.9749279121818236; case 11: return 0.9195277725514507; case 12:
        return 0.8345732537213026; case 13: return 0.7227948638273916; case 14: return 0.5877852522924731; case 15:
        return 0.4338837391175581; case 16: return 0.2660368455666751; case 17: return 0.0896393089034335; default:
        return 0; }
    } else if constexpr (R == 36) {
        switch (k) { case 0: return 0.0; case 1: return 0.17364817766693036; case 2: return 0.3420201433256687; case
        3: return 0.5; case 4: return 0.6427876096865394; case 5: return 0.766044443118978; case 6: return
        0.8660254037844386; case 7: return 0.9396926207859084; case 8: return 0.984807753012208; case 9: return 1.0;
        case 10: return 0.984807753012208; case 11: return 0.9396926207859084; case 12: return 0.8660254037844386;
        case 13: return 0.766044443118978; case 14: return 0.6427876096865394; case 15: return 0.5; case 16: return
        0.3420201433256687; case 17: return 0.17364817766693036; case 18: return 0.0; default: return 0; }
    }
    return 0;
}

template <int R> __device__ constexpr double root_cos(int k) { return root_cos_half<R>(2 * k <= R ? k : R - k); }
template <int R> __device__ constexpr double root_sin(int k) {
    return 2 * k <= R ? root_sin_half<R>(k) : -root_sin_half<R>(R - k);
}

// Odd prime length by its definition, the conjugate pairs of inputs and outputs taken together:
// with t_k = v_k + v_(R-k), s_k = v_k - v_(R-k), X_q and X_(R-q) are
// v_0 + sum cos(2 pi q k / R) t_k -+ i sum sin(2 pi q k / R) s_k.
template <int R, bool INV, typename T2> __device__ __forceinline__ void codelet_prime(T2 (&v)[R]) {
    using S = decltype(v[0].x);
    constexpr int H = (R - 1) / 2;
    T2 t[H], s[H];
    T2 sum = v[0];
#pragma unroll
    for (int k = 0; k < H; ++k) {
        t[k] = cadd(v[k + 1], v[R - 1 - k]);
        s[k] = csub(v[k + 1], v[R - 1 - k]);
        sum = cadd(sum, t[k]);
    }
    const T2 v0 = v[0];
    v[0] = sum;
#pragma unroll
    for (int q = 1; q <= H; ++q) {
        T2 a = v0, b = czero<T2>();
#pragma unroll
        for (int k = 0; k < H; ++k) {
            const int e = q * (k + 1) % R;
            const S c = (S)root_cos<R>(e), d = (S)root_sin<R>(e);
            a.x += c * t[k].x;
            a.y += c * t[k].y;
            b.x += d * s[k].x;
            b.y += d * s[k].y;
        }
        b = rot<INV>(b);
        v[q] = cadd(a, b);
        v[R - q] = csub(a, b);
    }
}

template <int R, bool INV, typename T2> __device__ __forceinline__ void codelet(T2 (&v)[R]);

// R = A B: B transforms of A points over v[b + B a], twiddles w_R^(b ka), A transforms of B points.
template <int A, int B, bool INV, typename T2> __device__ __forceinline__ void codelet_split(T2 (&v)[A * B]) {
    using S = decltype(v[0].x);
    constexpr int R = A * B;
    T2 u[B][A];
#pragma unroll
    for (int b = 0; b < B; ++b) {
#pragma unroll
        for (int a = 0; a < A; ++a) u[b][a] = v[b + B * a];
        codelet<A, INV>(u[b]);
#pragma unroll
        for (int a = 1; a < A; ++a)
            if (b) u[b][a] = twc<INV>(u[b][a], (S)root_cos<R>(a * b), (S)-root_sin<R>(a * b));
    }
#pragma unroll
    for (int a = 0; a < A; ++a) {
        T2 w[B];
#pragma unroll
        for (int b = 0; b < B; ++b) w[b] = u[b][a];
        codelet<B, INV>(w);
#pragma unroll
        for (int b = 0; b < B; ++b) v[a + A * b] = w[b];
    }
}

template <int R, bool INV, typename T2> __device__ __forceinline__ void codelet(T2 (&v)[R]) {
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        dft2<INV>(v[0], v[1]);
    } else if constexpr (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        dft8<INV>(v);
    } else if constexpr (R == 16) {
        dft16<INV>(v);
    } else if constexpr (R == 3 || R == 5 || R == 7) {
        codelet_prime<R, INV>(v);
    } else if constexpr (R == 9) {
        codelet_split<3, 3, INV>(v);
    } else if constexpr (R % 8 == 0) {
        codelet_split<8, R / 8, INV>(v);
    } else if constexpr (R % 4 == 0) {
        codelet_split<4, R / 4, INV>(v);
    } else if constexpr (R % 9 == 0) {
        codelet_split<9, R / 9, INV>(v);
    } else if constexpr (R % 5 == 0) {
        codelet_split<5, R / 5, INV>(v);
    } else if constexpr (R % 7 == 0) {
        codelet_split<7, R / 7, INV>(v);
    } else {
        codelet_split<3, R / 3, INV>(v);
    }
}

// ---------------------------------------------------------------------------------------------
// Codelet lengths by register class: class 0 for n1 <= 16, class 1 up to 36.
template <int N> using Len = std::integral_constant<int, N>;
template <int CLS, class F> __device__ __forceinline__ void with_n1(int n1, F&& f) {
    if constexpr (CLS == 0) {
        switch (n1) {
            case 4: f(Len<4>{}); break;
            case 5: f(Len<5>{}); break;
            case 6: f(Len<6>{}); break;
            case 7: f(Len<7>{}); break;
            case 8: f(Len<8>{}); break;
            case 9: f(Len<9>{}); break;
            case 10: f(Len<10>{}); break;
            case 12: f(Len<12>{}); break;
            case 14: f(Len<14>{}); break;
            case 15: f(Len<15>{}); break;
            default: f(Len<16>{}); break;
        }
    } else {
        switch (n1) {
            case 18: f(Len<18>{}); break;
            case 20: f(Len<20>{}); break;
            case 21: f(Len<21>{}); break;
            case 24: f(Len<24>{}); break;
            case 25: f(Len<25>{}); break;
            case 27: f(Len<27>{}); break;
            case 28: f(Len<28>{}); break;
            case 30: f(Len<30>{}); break;
            case 32: f(Len<32>{}); break;
            case 35: f(Len<35>{}); break;
            default: f(Len<36>{}); break;
        }
    }
}
template <int CLS, class F> __device__ __forceinline__ void with_n2(int n2, F&& f) {
    if constexpr (CLS == 0) {
        switch (n2) {
            case 3: f(Len<3>{}); break;
            case 4: f(Len<4>{}); break;
            case 5: f(Len<5>{}); break;
            case 6: f(Len<6>{}); break;
            case 7: f(Len<7>{}); break;
            case 8: f(Len<8>{}); break;
            case 9: f(Len<9>{}); break;
            case 10: f(Len<10>{}); break;
            case 12: f(Len<12>{}); break;
            case 14: f(Len<14>{}); break;
            case 15: f(Len<15>{}); break;
            default: f(Len<16>{}); break;
        }
    } else {
        switch (n2) {
            case 5: f(Len<5>{}); break;
            case 7: f(Len<7>{}); break;
            case 9: f(Len<9>{}); break;
            case 10: f(Len<10>{}); break;
            case 14: f(Len<14>{}); break;
            case 15: f(Len<15>{}); break;
            case 16: f(Len<16>{}); break;
            case 18: f(Len<18>{}); break;
            case 20: f(Len<20>{}); break;
            case 21: f(Len<21>{}); break;
            case 24: f(Len<24>{}); break;
            case 25: f(Len<25>{}); break;
            case 27: f(Len<27>{}); break;
            case 28: f(Len<28>{}); break;
            case 30: f(Len<30>{}); break;
            default: f(Len<32>{}); break;
        }
    }
}

// Threads of a CTA at most, and CTAs an SM its registers are sized for (FP64 class 1: 168 registers, class 0:
// 128; FP32: 128 and 80).
template <typename T, int CLS> struct RegShape {
    static constexpr int threads = sizeof(T) == 8 ? (CLS ? 192 : 128) : 256;
    static constexpr int blocks = sizeof(T) == 8 ? (CLS ? 2 : 4) : (CLS ? 2 : 3);
};

// The tables of a plan in the precision of T2: roots of length m, chirp (n) and kernel spectrum (m) of a
// Bluestein plan.
template <typename T2> struct RegTables;
template <> struct RegTables<double2> {
    __device__ static const double2* roots(const RegPlan& p) { return p.tw64; }
    __device__ static const double2* chirp(const RegPlan& p) { return p.chirp64; }
    __device__ static const double2* kern(const RegPlan& p) { return p.kern64; }
};
template <> struct RegTables<float2> {
    __device__ static const float2* roots(const RegPlan& p) { return p.tw32; }
    __device__ static const float2* chirp(const RegPlan& p) { return p.chirp32; }
    __device__ static const float2* kern(const RegPlan& p) { return p.kern32; }
};

// A line's buffer of n1 rows and n2 columns: element (r, c) at base[r rs + c cs].
template <typename T2> struct RegLine {
    T2* base;
    int rs, cs;
    __device__ __forceinline__ T2& at(int r, int c) const { return base[r * rs + c * cs]; }
};

// A layout to the buffer: thread t < n2 with v[m1] = x[n2 m1 + t]. Only thread t touches column t.
template <int R, typename T2>
__device__ __forceinline__ void reg_a_fwd(T2 (&v)[R], int t, const T2* __restrict__ tw, const RegLine<T2>& l) {
    codelet<R, false>(v);
#pragma unroll
    for (int k1 = 0; k1 < R; ++k1) l.at(k1, t) = k1 ? cmul(v[k1], __ldg(&tw[t * k1])) : v[k1];
}
// The buffer to the B layout: thread k1 < n1, v[k2] = X[k1 + n1 k2]. Only thread k1 touches row k1.
template <int R, typename T2> __device__ __forceinline__ void reg_b_fwd(T2 (&v)[R], int k1, const RegLine<T2>& l) {
#pragma unroll
    for (int c = 0; c < R; ++c) v[c] = l.at(k1, c);
    codelet<R, false>(v);
}
template <int R, typename T2>
__device__ __forceinline__ void reg_b_inv(T2 (&v)[R], int k1, const T2* __restrict__ tw, const RegLine<T2>& l) {
    codelet<R, true>(v);
#pragma unroll
    for (int c = 0; c < R; ++c) l.at(k1, c) = c ? cmulc(v[c], __ldg(&tw[c * k1])) : v[c];
}
// v[m1] = m x[n2 m1 + t] (unnormalised).
template <int R, typename T2> __device__ __forceinline__ void reg_a_inv(T2 (&v)[R], int t, const RegLine<T2>& l) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = l.at(r, t);
    codelet<R, true>(v);
}

// The middle of a Bluestein transform, between the buffer's A side and its A side: the convolution with the
// chirp's kernel (its conjugate for the inverse). Starts and ends with a barrier.
template <int CLS, bool INV, typename T2>
__device__ __forceinline__ void reg_convolve(const RegPlan& p, int t, bool on, const RegLine<T2>& l) {
    const T2* kern = RegTables<T2>::kern(p);
    const T2* tw = RegTables<T2>::roots(p);
    __syncthreads();
    with_n2<CLS>(p.n2, [&](auto len) {
        constexpr int R = decltype(len)::value;
        if (on && t < p.n1) {
            T2 v[R];
            reg_b_fwd<R>(v, t, l);
#pragma unroll
            for (int k2 = 0; k2 < R; ++k2) {
                const T2 w = __ldg(&kern[t + p.n1 * k2]);
                v[k2] = INV ? cmulc(v[k2], w) : cmul(v[k2], w);
            }
            reg_b_inv<R>(v, t, tw, l);
        }
    });
    __syncthreads();
}

}  // namespace rtm
